// vc1cu_global.cu - whole-frame translation search, Vc1Encoder::global_motion_search and
// global_motion_search_extended (encoder_motion.cpp:2025-2141), for many pictures at once.
//
// Each stage of the reference is a fixed candidate list (given the previous stage) scored
// with frame_sad (encoder_motion.cpp:1499-1576) and then folded by a sequential rule
// (top-8 insertion with truncation, first-visit tie breaks). Here every stage is one
// parallel scoring launch (one block per candidate x row slab, partial sums combined with
// integer atomics, so the order of summation does not matter); the last block of a picture to
// finish folds the stage's costs and plans the next stage, so a search is one planning launch
// and one launch per stage.
//
// The fold is bound by latency, not work (at most 392 costs per stage). Its rules are restated
// in an order-free form where the reference's result is one: the plain search's top-8 insertion
// with truncation keeps the eight least of a multiset, found by ranking every cost against every
// other; its refinement keeps the first-visited least cost, a minimum over (cost, |d|, slot) with
// the visit order as the slot index. The extended search's list (least cost per vector, sorted
// only on insertion) does depend on the order and is replayed by one warp, entry per lane.
// Folding on one thread, with the lists in global memory, took 0.87 ms of a CIF search, 2.3 ms of two
// at 1080p; folded here it is within the scoring launches' time.
#include <cuda.h>  // CUcontext (cuCtxGetId is reached through the runtime's entry point)
#include <cuda_runtime.h>

#include <cstdio>
#include <map>
#include <mutex>

#include "vc1cu_core.cuh"

namespace vc1cu {

constexpr int kGMaxCand = 512;  // largest stage: range 31 refine, 8 x 7 x 7 = 392
constexpr int kGThreads = 256;
constexpr int kGTop = 8;

// One search's inputs and output addresses.
struct GIn {
    DevFrame cur, ref;
    int range;                 // min(local range, 32)
    int* out_global;           // [dx, dy]
    unsigned long long* out_sad;
};

struct GState {
    GIn in;
    int n;                     // candidate slots of the current stage
    int arrived;               // blocks of the current stage that have finished
    int top_n;
    int sorted;                // extended search: no cost was lowered since the list's last insertion
    int2 top[kGTop];
    unsigned long long top_cost[kGTop];
    int2 cand[kGMaxCand];      // x = INT_MIN: an empty slot
    unsigned long long cost[kGMaxCand];
};

constexpr int kGEmpty = -0x7fffffff - 1;

// (cost, |dx| + |dy|, dy, dx) in one comparable key: a frame SAD of at most 16384 x 16384 samples
// is below 2^37, |d| <= 64 and each component within [-32, 32].
__device__ __forceinline__ unsigned long long gkey(unsigned long long cost, int2 d) {
    return (cost << 21) | ((unsigned long long)(iabs(d.x) + iabs(d.y)) << 14) | ((unsigned long long)(d.y + 32) << 7) |
           (unsigned long long)(d.x + 32);
}

// Sampling stride of a search's stages.
__host__ __device__ inline int gstage_stride(int R, int stage) {
    if (R <= 0) return 1;
    if (R <= 31) return stage == 0 ? 4 : (stage == 1 ? 2 : 1);
    return stage == 0 ? 16 : (stage == 1 ? 8 : (stage == 2 ? 4 : 1));
}
__host__ __device__ inline int gstage_count(int R) { return R <= 0 ? 1 : (R <= 31 ? 3 : 4); }
__host__ __device__ inline int gcoarse_step(int R) { return R >= 4 ? 4 : (R >= 2 ? 2 : 1); }
constexpr int kGExtStep = 8;  // the extended search's step (its range is 32 here)

// Candidate slots of a stage (an upper bound where slots may be empty).
__host__ __device__ inline int gstage_slots(int R, int stage) {
    if (R <= 0) return 1;
    if (R <= 31) {
        const int cs = gcoarse_step(R), L = (2 * R) / cs + 1, w = 2 * cs - 1;
        return stage == 0 ? L * L + 1 + 2 * L : (stage == 1 ? kGTop * w * w : 1);
    }
    const int k = R / kGExtStep, g = (2 * kGExtStep) / 4 + 1;
    return stage == 0 ? 1 + 12 * k : (stage == 1 ? 4 * g * g : (stage == 2 ? 81 : 9));
}

// Slot t of a search's first stage: the coarse grid, zero and the far edges (:2110-2124), or the
// extended search's cross and octagon rings (:2040-2052).
__device__ __forceinline__ int2 gfirst(int R, int t) {
    if (R <= 0) return make_int2(0, 0);
    if (R <= 31) {
        const int cs = gcoarse_step(R), L = (2 * R) / cs + 1;
        if (t < L * L) return make_int2(-R + (t % L) * cs, -R + (t / L) * cs);
        if (t == L * L) return make_int2(0, 0);
        const int j = t - L * L - 1, d = -R + (j >> 1) * cs;
        return (j & 1) ? make_int2(d, R) : make_int2(R, d);
    }
    if (t == 0) return make_int2(0, 0);
    const int k = R / kGExtStep;
    int2 v;
    if (t <= 4 * k) {
        const int d = kGExtStep * ((t - 1) / 4 + 1), a = (t - 1) & 3;
        v = a == 0 ? make_int2(-d, 0) : a == 1 ? make_int2(d, 0) : a == 2 ? make_int2(0, -d) : make_int2(0, d);
    } else {
        const int j = t - 1 - 4 * k, r = kGExtStep * (j / 8 + 1), h = (r + 1) / 2, a = j & 7;
        // (-r,-h) (-r,h) (r,-h) (r,h) (-h,-r) (h,-r) (-h,r) (h,r)
        v = a < 4 ? make_int2(a < 2 ? -r : r, (a & 1) ? h : -h) : make_int2((a & 1) ? h : -h, a < 6 ? -r : r);
    }
    return make_int2(iclamp(v.x, -R, R), iclamp(v.y, -R, R));
}

// One block per search: takes its inputs (when given) and lays out the first stage.
__global__ void __launch_bounds__(kGThreads) gplan_kernel(GState* states, const GIn* in) {
    GState& s = states[blockIdx.x];
    const int R = in ? in[blockIdx.x].range : s.in.range;
    const int n = gstage_slots(R, 0);
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        s.cand[t] = gfirst(R, t);
        s.cost[t] = 0;
    }
    if (threadIdx.x == 0) {
        if (in) s.in = in[blockIdx.x];
        s.n = n;
        s.arrived = 0;
        s.top_n = 0;
        s.sorted = 1;
    }
}

// The least `v` of the block, on every thread.
__device__ unsigned long long block_min(unsigned long long v, unsigned long long* red) {
    v = warp_min_u64(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = red[w] < v ? red[w] : v;
    return v;
}

// `consider` of global_motion_search_extended (:2034-2039) over the stage's costs, by warp 0:
// lane i holds list entry i (the entry's own vector once, its least cost; sorted by insertion, so
// a lowered cost stays in place until the next insertion, then the eight least are kept).
__device__ void gfold_ext(GState& s, const unsigned long long* cost, int n, unsigned long long* red) {
    const int lane = threadIdx.x;
    if (lane >= 32) return;
    int tn = s.top_n;
    int2 v = lane < tn ? s.top[lane] : make_int2(0, 0);
    unsigned long long c = lane < tn ? s.top_cost[lane] : 0;
    bool sorted = s.sorted != 0;
    for (int k = 0; k < n; ++k) {
        const int2 q = s.cand[k];
        const unsigned long long qc = cost[k];
        const bool hit = lane < tn && v.x == q.x && v.y == q.y;
        if (__any_sync(0xffffffffu, hit)) {
            const bool lower = hit && qc < c;
            if (lower) c = qc;
            if (__any_sync(0xffffffffu, lower)) sorted = false;
            continue;
        }
        const unsigned long long last = __shfl_sync(0xffffffffu, gkey(c, v), kGTop - 1);
        if (sorted && tn == kGTop && gkey(qc, q) > last) continue;  // would be inserted last and cut
        if (lane == tn) {
            v = q;
            c = qc;
        }
        ++tn;
        const unsigned long long mine = gkey(c, v);
        int rank = 0;
        for (int j = 0; j < tn; ++j) rank += __shfl_sync(0xffffffffu, mine, j) < mine ? 1 : 0;
        // entries move to their ranks through shared memory
        if (lane < tn) {
            red[2 * rank] = c;
            red[2 * rank + 1] = ((unsigned long long)(uint32_t)v.x << 32) | (uint32_t)v.y;
        }
        __syncwarp();
        if (lane < tn) {
            c = red[2 * lane];
            const unsigned long long p = red[2 * lane + 1];
            v = make_int2((int)(uint32_t)(p >> 32), (int)(uint32_t)p);
        }
        __syncwarp();
        tn = imin(tn, kGTop);
        sorted = true;
    }
    if (lane < tn) {
        s.top[lane] = v;
        s.top_cost[lane] = c;
    }
    if (lane == 0) {
        s.top_n = tn;
        s.sorted = sorted ? 1 : 0;
    }
}

// Folds the finished stage's costs and lays out the next stage (or writes the result); one block.
__device__ void gfold(GState& s, int stage) {
    __shared__ unsigned long long key[kGMaxCand];
    __shared__ unsigned long long red[32];
    const int R = s.in.range, n = s.n, st = gstage_stride(R, stage);
    const unsigned long long scale = (unsigned long long)(st * st);
    const bool plain = R <= 31;
    __syncthreads();
    if (plain && stage == 0 && R > 0) {
        // the eight least of (cost, |d|, dy, dx), repeats kept (:2086-2098)
        for (int t = threadIdx.x; t < n; t += blockDim.x) key[t] = gkey(__ldcg(&s.cost[t]) * scale, s.cand[t]);
        __syncthreads();
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const unsigned long long k = key[t];
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += (key[j] < k || (key[j] == k && j < t)) ? 1 : 0;
            if (rank < kGTop) s.top[rank] = s.cand[t];
        }
        __syncthreads();
        // the refinement's visit list (:2129-2140): a window about each entry, first visits only
        const int cs = gcoarse_step(R), w = 2 * cs - 1, tn = imin(kGTop, n), m = tn * w * w;
        int2 top[kGTop];
#pragma unroll
        for (int k = 0; k < kGTop; ++k) top[k] = k < tn ? s.top[k] : make_int2(0, 0);
        for (int t = threadIdx.x; t < m; t += blockDim.x) {
            const int k = t / (w * w), q = t - k * w * w;
            const int2 c0 = s.top[k];
            int2 d = make_int2(c0.x - (cs - 1) + q % w, c0.y - (cs - 1) + q / w);
            bool ok = iabs(d.x) <= R && iabs(d.y) <= R;
#pragma unroll
            for (int j = 0; j < kGTop; ++j)
                if (j < k && iabs(d.x - top[j].x) < cs && iabs(d.y - top[j].y) < cs) ok = false;
            if (!ok) d.x = kGEmpty;
            s.cand[t] = d;
            s.cost[t] = 0;
        }
        if (threadIdx.x == 0) s.n = m;
        return;
    }
    if (plain && stage == 1) {
        // the first-visited least (cost, |d|) (:2129-2140)
        unsigned long long best = ~0ull;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int2 d = s.cand[t];
            if (d.x == kGEmpty) continue;
            const unsigned long long k = ((__ldcg(&s.cost[t]) * scale) << 16) |
                                         ((unsigned long long)(iabs(d.x) + iabs(d.y)) << 9) | (unsigned long long)t;
            best = k < best ? k : best;
        }
        best = block_min(best, red);
        if (threadIdx.x == 0) {
            const int2 d = s.cand[(int)(best & 511)];
            s.cand[0] = d;
            s.cost[0] = 0;
            s.n = 1;
        }
        return;
    }
    if (plain) {
        // range 0: frame_sad(0, 0, 1) (:2082-2085); else the chosen vector's full frame SAD
        if (threadIdx.x == 0) {
            const int2 d = s.cand[0];
            s.in.out_global[0] = d.x;
            s.in.out_global[1] = d.y;
            *s.in.out_sad = __ldcg(&s.cost[0]);
        }
        return;
    }
    if (stage < 3) {
        for (int t = threadIdx.x; t < n; t += blockDim.x) key[t] = __ldcg(&s.cost[t]) * scale;
        __syncthreads();
        gfold_ext(s, key, n, red);
        __syncthreads();
        // stage 1: 5x5 at step 4 about the four best; stages 2 and 3: 9x9 and 3x3 about the best
        const int g = stage == 0 ? (2 * kGExtStep) / 4 + 1 : (stage == 1 ? 9 : 3);
        const int step = stage == 0 ? 4 : 1, nc = stage == 0 ? imin(4, s.top_n) : 1, m = nc * g * g;
        for (int t = threadIdx.x; t < m; t += blockDim.x) {
            const int2 c0 = s.top[t / (g * g)];
            const int q = t % (g * g), h = step * (g / 2);
            s.cand[t] = make_int2(iclamp(c0.x - h + step * (q % g), -R, R), iclamp(c0.y - h + step * (q / g), -R, R));
            s.cost[t] = 0;
        }
        if (threadIdx.x == 0) s.n = m;
        return;
    }
    // the full-resolution 3x3: least by the total order (:2066-2074)
    unsigned long long best = ~0ull;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const unsigned long long k = gkey(__ldcg(&s.cost[t]), s.cand[t]);
        best = k < best ? k : best;
    }
    best = block_min(best, red);
    if (threadIdx.x == 0) {
        s.in.out_global[0] = (int)(best & 127) - 32;
        s.in.out_global[1] = (int)((best >> 7) & 127) - 32;
        *s.in.out_sad = best >> 21;
    }
}

// frame_sad of every candidate of every search: grid (slab, candidate slot, search).
// Two 1080p searches at range 32 (8 launches, the folds included): 277 us, against 363 us for the
// scoring alone with one sample per load.
__global__ void __launch_bounds__(kGThreads) gsad_kernel(GState* states, int W, int H, int rows_per_slab, int stage) {
    GState& s = states[blockIdx.z];
    const int ci = blockIdx.y;
    const int st = gstage_stride(s.in.range, stage);
    const int nrows = (H + st - 1) / st, r0 = blockIdx.x * rows_per_slab, r1 = imin(nrows, r0 + rows_per_slab);
    const int2 c = ci < s.n ? s.cand[ci] : make_int2(kGEmpty, 0);
    const bool scored = c.x != kGEmpty && r0 < r1;
    __shared__ unsigned long long part[kGThreads / 32];
    if (scored) {
        const uint32_t acc = frame_sad_part(s.in.cur.y, s.in.cur.pitch_y, s.in.ref.y, s.in.ref.pitch_y, W, H, c.x, c.y, st, r0, r1);
        const uint64_t sum = warp_sum_u64(acc);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    }
    // Every warp has read its slot before the block counts as finished, an empty slot's too: the last
    // block rewrites the slots.
    __syncthreads();
    // the last block of this search to arrive sees every block's cost and folds the stage
    __shared__ bool last;
    if (threadIdx.x == 0) {
        if (scored) {
            unsigned long long t = 0;
            for (int w = 0; w < kGThreads / 32; ++w) t += part[w];
            atomicAdd(&s.cost[ci], t);
        }
        __threadfence();
        last = atomicAdd(&s.arrived, 1) == (int)(gridDim.x * gridDim.y) - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    gfold(s, stage);
    if (threadIdx.x == 0) s.arrived = 0;
}

size_t gstate_bytes() { return sizeof(GState); }
size_t gin_bytes() { return sizeof(GIn); }

// Passes that share one search take its result: one thread per copy (dx, dy and the SAD).
__global__ void global_fanout_kernel(const GlobalCopy* copies, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GlobalCopy c = copies[i];
    c.dst_global[0] = c.src_global[0];
    c.dst_global[1] = c.src_global[1];
    *c.dst_sad = *c.src_sad;
}

cudaError_t launch_global_fanout(const GlobalCopy* d_copies, int n, cudaStream_t s) {
    if (n > 0) global_fanout_kernel<<<(n + 127) / 128, 128, 0, s>>>(d_copies, n);
    return cudaGetLastError();
}

// Host driver: runs the staged search for n searches whose inputs are in device memory (d_in; or
// already in the states when d_in is null): a planning launch, then one launch per stage, sized
// to the stage's candidate slots and sampling stride. Returns the launches.
int run_global_search(GState* d_states, const GIn* d_in, int n, int R, int W, int H, cudaStream_t stream) {
    const int rows_per_slab = 64;
    gplan_kernel<<<n, kGThreads, 0, stream>>>(d_states, d_in);
    const int ns = gstage_count(R);
    for (int i = 0; i < ns; ++i) {
        const int st = gstage_stride(R, i), rows = (H + st - 1) / st;
        const dim3 grid((rows + rows_per_slab - 1) / rows_per_slab, gstage_slots(R, i), n);
        gsad_kernel<<<grid, kGThreads, 0, stream>>>(d_states, W, H, rows_per_slab, i);
    }
    return 1 + ns;
}

void init_gin(GIn* h, const DevFrame& cur, const DevFrame& ref, int range, int* out_global,
              unsigned long long* out_sad) {
    h->cur = cur;
    h->ref = ref;
    h->range = range;
    h->out_global = out_global;
    h->out_sad = out_sad;
}

// ---- allocation-free form (vc1cu_global_motion_noalloc) ---------------------------------
//
// Some callers cannot allocate device memory while they run: an encoder thread working out
// of a fixed device-memory budget, or code that runs where a cudaMalloc would synchronise
// the device or is not permitted. For them the search state of up to
// kNoAllocMaxPictures pictures lives in this fixed array, which every GPU that loads the
// library holds until the process exits (16 states of 8,424 bytes: 134,784 bytes).
// Every call shares it; calls are ordered on the device, one after another.
constexpr int kNoAllocMaxPictures = 16;
static __device__ __align__(256) GState g_noalloc_states[kNoAllocMaxPictures];
static_assert(sizeof(GState) * kNoAllocMaxPictures == 134784, "the size the interface documents");

struct NoAllocInit {
    DevFrame cur[kNoAllocMaxPictures], ref[kNoAllocMaxPictures];
    int* out_global;
    unsigned long long* out_sad;
    int range, n;
};

// Writes each search's inputs; the planning launch that follows resets all that a search reads,
// so a call never sees the previous call's state.
__global__ void noalloc_init_kernel(GState* states, const __grid_constant__ NoAllocInit a) {
    const int i = threadIdx.x;
    if (i >= a.n) return;
    GIn& s = states[i].in;
    s.cur = a.cur[i];
    s.ref = a.ref[i];
    s.range = a.range;
    s.out_global = a.out_global + 2 * i;
    s.out_sad = a.out_sad + i;
}

}  // namespace vc1cu

namespace {

// The order of the calls that share a context's array: each call's work waits for the event after the
// work of the call before it, whatever streams and threads they come from. One event per context (its
// id is never given again, so an event that went with its context is not used).
std::mutex& noalloc_mutex() {
    static std::mutex* m = new std::mutex;  // not destroyed: calls may come from exit handlers
    return *m;
}

cudaError_t noalloc_event(cudaEvent_t* e) {
    using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);
    static CtxGetIdFn ctx_id = []() -> CtxGetIdFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<CtxGetIdFn>(p);
    }();
    static auto* events = new std::map<unsigned long long, cudaEvent_t>;
    unsigned long long id = 0;
    if (!ctx_id || ctx_id(nullptr, &id) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
    cudaEvent_t& ev = (*events)[id];
    if (!ev) {
        const cudaError_t rc = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (rc != cudaSuccess) {
            events->erase(id);
            return rc;
        }
    }
    *e = ev;
    return cudaSuccess;
}

int noalloc_fail(char* err, size_t err_len, int code, const char* msg) {
    if (err && err_len) std::snprintf(err, err_len, "%s", msg);
    return code;
}

}  // namespace

extern "C" int vc1cu_global_motion_noalloc(const uint8_t* const* cur_y, const uint8_t* const* ref_y, int pitch,
                                           int width, int height, int range, int n, int32_t* d_dxdy,
                                           uint64_t* d_sad, void* stream, char* err, size_t err_len) {
    using namespace vc1cu;
    if (err && err_len) err[0] = 0;
    if (n < 1 || n > kNoAllocMaxPictures)
        return noalloc_fail(err, err_len, VC1CU_ERR_ARG,
                            "vc1cu_global_motion_noalloc: n must be 1..16 pictures per call (the fixed scratch size)");
    if (width <= 0 || height <= 0 || width > 16384 || height > 16384 || pitch < width)
        return noalloc_fail(err, err_len, VC1CU_ERR_ARG,
                            "vc1cu_global_motion_noalloc: width/height must be 1..16384 and pitch >= width");
    if (range < 0 || range > 32)
        return noalloc_fail(err, err_len, VC1CU_ERR_ARG, "vc1cu_global_motion_noalloc: range must be 0..32");
    if (!cur_y || !ref_y || !d_dxdy || !d_sad)
        return noalloc_fail(err, err_len, VC1CU_ERR_ARG, "vc1cu_global_motion_noalloc: null pointer argument");
    NoAllocInit a{};
    for (int i = 0; i < n; ++i) {
        if (!cur_y[i] || !ref_y[i])
            return noalloc_fail(err, err_len, VC1CU_ERR_ARG, "vc1cu_global_motion_noalloc: null frame pointer");
        a.cur[i] = DevFrame{cur_y[i], nullptr, nullptr, pitch, 0};
        a.ref[i] = DevFrame{ref_y[i], nullptr, nullptr, pitch, 0};
    }
    a.out_global = reinterpret_cast<int*>(d_dxdy);
    a.out_sad = reinterpret_cast<unsigned long long*>(d_sad);
    a.range = range;
    a.n = n;
    // The host-side name of a __device__ array is not a device address. The address is looked
    // up on every call, with the caller's device current, so it is always the one of the module
    // loaded in the current context (a cached value would dangle after cudaDeviceReset).
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_states);
    if (e != cudaSuccess || !ptr)
        return noalloc_fail(err, err_len, VC1CU_ERR_CUDA,
                            e != cudaSuccess ? cudaGetErrorString(e) : "cudaGetSymbolAddress returned null");
    GState* states = static_cast<GState*>(ptr);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // a captured call is ordered by whoever replays it
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess) return noalloc_fail(err, err_len, VC1CU_ERR_CUDA, cudaGetErrorString(e));
    std::lock_guard<std::mutex> lock(noalloc_mutex());
    cudaEvent_t after = nullptr;
    if (capture == cudaStreamCaptureStatusNone) {
        e = noalloc_event(&after);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, after, 0);
        if (e != cudaSuccess) return noalloc_fail(err, err_len, VC1CU_ERR_CUDA, cudaGetErrorString(e));
    }
    noalloc_init_kernel<<<1, 32, 0, s>>>(states, a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return noalloc_fail(err, err_len, VC1CU_ERR_CUDA, cudaGetErrorString(e));
    run_global_search(states, nullptr, n, range, width, height, s);
    e = cudaGetLastError();
    if (after) {
        const cudaError_t r = cudaEventRecord(after, s);
        if (e == cudaSuccess) e = r;
    }
    if (e != cudaSuccess) return noalloc_fail(err, err_len, VC1CU_ERR_CUDA, cudaGetErrorString(e));
    return VC1CU_OK;
}
