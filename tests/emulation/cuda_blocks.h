// Runs CUDA kernels' source on the host, every thread of a launch as a coroutine, so that a test can
// choose the order in which the warps of different blocks advance. A block barrier that the threads of
// a block meet at different source lines, and threads that wait for one another for good, are
// recorded as faults. The source is compiled with __shared__ declarations and <<< >>> launches
// rewritten to emu::shared and EMU_LAUNCH (see test_global_search_blocks.py).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <string>
#include <tuple>
#include <vector>

#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __grid_constant__
#define __grid_constant__

namespace emu {

struct Block;

struct Thread {
    enum State { kReady, kBarrier, kWarp, kDone };
    ucontext_t ctx;
    Block* block = nullptr;
    unsigned tid = 0;
    State state = kReady;
    int line = 0;     // of the barrier waited at
    int ops = 0;      // warp exchanges entered
    bool begun = false;
};

struct Block {
    dim3 idx;
    std::vector<Thread> threads;
    std::vector<uint64_t> lanes[2];  // warp exchange values, by the parity of the exchange
    std::map<const void*, std::unique_ptr<uint64_t[]>> shared;
    int live = 0;
    size_t begun = 0;  // threads that have run at all
};

// Which thread runs next. kInOrder: by block, then by thread. kLateWarps: the first warp of every
// block first; then the blocks whose first warp waits at the earliest barrier; of those that wait at
// the same one, the blocks whose other warps have begun. So the warps of a block whose first warp met
// no barrier on its way begin after everyone else's have ended.
enum Order { kInOrder, kLateWarps };

inline Thread* cur = nullptr;
inline ucontext_t scheduler;
inline dim3 grid_dim, block_dim;
inline const std::function<void()>* body = nullptr;
inline Order order = kInOrder;
inline std::string fault;
inline std::vector<std::string> trace;  // launches ("launch <stream>"), and what the test's stubs add

inline void yield(Thread::State s) {
    Thread* t = cur;
    t->state = s;
    swapcontext(&t->ctx, &scheduler);
}

inline void trampoline() {
    (*body)();
    cur->state = Thread::kDone;
    --cur->block->live;
    swapcontext(&cur->ctx, &scheduler);
}

inline void syncthreads(int line) {
    cur->line = line;
    yield(Thread::kBarrier);
}

// Every lane of the warp puts in a value; the returned array holds all 32.
inline const uint64_t* exchange(uint64_t v) {
    auto& buf = cur->block->lanes[cur->ops++ & 1];
    buf[cur->tid] = v;
    yield(Thread::kWarp);
    return &buf[cur->tid & ~31u];
}

template <class T, int LINE>
T& shared() {
    static const char key = 0;
    auto& p = cur->block->shared[&key];
    if (!p) {
        p.reset(new uint64_t[(sizeof(T) + 7) / 8]);
        std::memset(p.get(), 0xA5, sizeof(T));
    }
    return *reinterpret_cast<T*>(p.get());
}

// Releases the block's barrier or a warp's exchange once everyone who must take part waits there.
inline void release(Block& b, unsigned warp) {
    auto first = b.threads.begin() + 32 * warp, last = b.threads.begin() + std::min<size_t>(32 * warp + 32, b.threads.size());
    if (std::all_of(first, last, [](const Thread& t) { return t.state == Thread::kWarp; }))
        std::for_each(first, last, [](Thread& t) { t.state = Thread::kReady; });
    int line = 0, waiting = 0;
    bool same = true;
    for (const Thread& t : b.threads)
        if (t.state == Thread::kBarrier) {
            same = same && (!waiting || t.line == line);
            line = t.line;
            ++waiting;
        }
    if (!waiting || waiting != b.live) return;
    if (!same && fault.empty())
        fault = "block (" + std::to_string(b.idx.x) + ", " + std::to_string(b.idx.y) + "): its threads meet at different barriers";
    for (Thread& t : b.threads)
        if (t.state == Thread::kBarrier) t.state = Thread::kReady;
}

inline Thread* pick(std::vector<Block>& blocks) {
    Thread* best = nullptr;
    std::tuple<int, int, size_t> best_key;
    for (Block& b : blocks) {
        if (!b.live) continue;
        for (size_t i = 0; i < b.threads.size(); ++i) {
            Thread& t = b.threads[i];
            if (t.state != Thread::kReady) continue;
            if (order == kInOrder) return &t;
            const std::tuple<int, int, size_t> key{i < 32 ? 0 : 1, i < 32 ? 0 : b.threads[0].line,
                                                   i < 32 ? 0 : b.threads.size() - b.begun};
            if (!best || key < best_key) {
                best = &t;
                best_key = key;
            }
            if (i >= 32) break;  // the block's other threads have the same key
        }
        if (best && std::get<0>(best_key) == 0) return best;
    }
    return best;
}

struct Cfg {
    dim3 grid, block;
    cudaStream_t stream;
    Cfg(dim3 g, dim3 b, size_t = 0, cudaStream_t s = nullptr) : grid(g), block(b), stream(s) {}
    void run(const std::function<void()>& f) const {
        trace.push_back("launch " + std::to_string(reinterpret_cast<uintptr_t>(stream)));
        if (!fault.empty()) return;
        constexpr size_t kStack = 64 << 10;
        const size_t per = block.x, n = (size_t)grid.x * grid.y * grid.z;
        char* stacks = static_cast<char*>(mmap(nullptr, n * per * kStack, PROT_READ | PROT_WRITE,
                                               MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
        grid_dim = grid;
        block_dim = block;
        body = &f;
        std::vector<Block> blocks(n);
        for (size_t k = 0; k < n; ++k) {
            Block& b = blocks[k];
            b.idx = dim3((unsigned)(k % grid.x), (unsigned)(k / grid.x % grid.y), (unsigned)(k / grid.x / grid.y));
            b.threads.resize(per);
            b.live = (int)per;
            b.lanes[0].resize((per + 31) & ~size_t(31));
            b.lanes[1].resize((per + 31) & ~size_t(31));
            for (size_t i = 0; i < per; ++i) {
                Thread& t = b.threads[i];
                t.block = &b;
                t.tid = (unsigned)i;
                getcontext(&t.ctx);
                t.ctx.uc_stack.ss_sp = stacks + (k * per + i) * kStack;
                t.ctx.uc_stack.ss_size = kStack;
                t.ctx.uc_link = nullptr;
                makecontext(&t.ctx, trampoline, 0);
            }
        }
        while (Thread* t = pick(blocks)) {
            cur = t;
            if (!t->begun) {
                t->begun = true;
                ++t->block->begun;
            }
            swapcontext(&scheduler, &t->ctx);
            release(*t->block, t->tid / 32);
            if (!fault.empty()) break;
        }
        for (const Block& b : blocks)
            if (b.live && fault.empty()) fault = "threads of a block wait for one another";
        munmap(stacks, n * per * kStack);
    }
};

}  // namespace emu

#define EMU_LAUNCH(cfg, kernel, ...) emu::Cfg cfg.run([&] { kernel(__VA_ARGS__); })
#define threadIdx (dim3(emu::cur->tid, 0, 0))
#define blockIdx (emu::cur->block->idx)
#define gridDim emu::grid_dim
#define blockDim emu::block_dim
#define __syncthreads() emu::syncthreads(__LINE__)

inline void __threadfence() {}
inline void __syncwarp(unsigned = 0) { emu::exchange(0); }
template <class T> inline T __ldg(const T* p) { return *p; }
template <class T> inline T __ldcg(const T* p) { return *p; }
template <class T, class U> inline T atomicAdd(T* p, U v) { const T o = *p; *p = o + (T)v; return o; }

template <class T> inline T __shfl_sync(unsigned, T v, int lane) {
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof v);
    const uint64_t r = emu::exchange(b)[lane & 31];
    std::memcpy(&v, &r, sizeof v);
    return v;
}
template <class T> inline T __shfl_xor_sync(unsigned m, T v, int o) { return __shfl_sync(m, v, (int)(emu::cur->tid & 31) ^ o); }
inline int __any_sync(unsigned, int p) {
    const uint64_t* v = emu::exchange(p ? 1 : 0);
    return std::any_of(v, v + 32, [](uint64_t x) { return x != 0; });
}
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
inline unsigned __byte_perm(unsigned a, unsigned b, unsigned s) {
    const uint64_t v = ((uint64_t)b << 32) | a;
    unsigned r = 0;
    for (int i = 0; i < 4; ++i) r |= (unsigned)((v >> (8 * ((s >> (4 * i)) & 7))) & 255) << (8 * i);
    return r;
}
inline unsigned __vsadu4(unsigned a, unsigned b) {
    unsigned r = 0;
    for (int i = 0; i < 32; i += 8) r += (unsigned)std::abs((int)((a >> i) & 255) - (int)((b >> i) & 255));
    return r;
}
