"""The global translation search's kernels run on the host, thread by thread, under chosen orders.

A stage's last block to finish folds its costs and rewrites the candidate list that every block of
the stage has read. So no warp may still have its candidate to read once its block counts as
finished, however late that warp runs: the order "late warps" lets the first warp of each block run
ahead and holds the rest of a finished block back until nothing else can advance. The kernels'
source itself is compiled (emulation/cuda_blocks.h); the results are the oracle's.

The allocation-free form keeps its state in one array per device: a call's work has to wait for the
work of the call before it, whatever their streams.
"""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

from libvc1_b200.abi import make_params

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "libvc1_b200", "csrc")

MAIN = r"""
extern "C" int emulate(const uint8_t* cur, const uint8_t* ref, int w, int h, int range, int order, int* dxdy,
                       unsigned long long* sad, char* why, size_t cap) {
    emu::order = static_cast<emu::Order>(order);
    emu::fault.clear();
    const int rc = vc1cu_global_motion_noalloc(&cur, &ref, w, w, h, range, 1, dxdy, (uint64_t*)sad, nullptr, why, cap);
    if (!emu::fault.empty()) std::snprintf(why, cap, "%s", emu::fault.c_str());
    return rc ? rc : (emu::fault.empty() ? 0 : -1);
}
static bool g_capturing;
static std::string num(const void* p) { return std::to_string(reinterpret_cast<uintptr_t>(p)); }
// One call per stream; the launches, event records and waits that they make, one per line.
extern "C" int emulate_calls(const uint8_t* a, const uint8_t* b, int w, int h, const uintptr_t* streams, int n,
                             int capturing, char* out, size_t cap) {
    emu::order = emu::kInOrder;
    emu::fault.clear();
    emu::trace.clear();
    g_capturing = capturing != 0;
    int dxdy[2], rc = 0;
    uint64_t sad;
    for (int i = 0; i < n && !rc; ++i)
        rc = vc1cu_global_motion_noalloc(&a, &b, w, w, h, 1, 1, dxdy, &sad, reinterpret_cast<void*>(streams[i]), out, cap);
    std::string t;
    for (const auto& l : emu::trace) t += l + "\n";
    std::snprintf(out, cap, "%s", t.c_str());
    g_capturing = false;
    return rc;
}
static CUresult fake_ctx_id(CUcontext, unsigned long long* id) { *id = 7; return CUDA_SUCCESS; }
extern "C" cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long,
                                               cudaDriverEntryPointQueryResult* q) {
    *fn = reinterpret_cast<void*>(&fake_ctx_id);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
extern "C" cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
    *c = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
extern "C" cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    static uintptr_t next = 100;
    *e = reinterpret_cast<cudaEvent_t>(next++);
    return cudaSuccess;
}
extern "C" cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    emu::trace.push_back("wait " + num(s) + " " + num(e));
    return cudaSuccess;
}
extern "C" cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    emu::trace.push_back("record " + num(s) + " " + num(e));
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "emulated"; }
extern "C" cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
"""


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    d = tmp_path_factory.mktemp("blocks")
    src = open(os.path.join(CSRC, "vc1cu_global.cu")).read()
    src = re.sub(r"__shared__\s+([\w ]+?)\s+(\w+)((?:\[[^\]]*\])?);", r"auto& \2 = emu::shared<\1\3, __LINE__>();", src)
    src = re.sub(r"(\w+)<<<([^;]*?)>>>\(([^;]*)\);", r"EMU_LAUNCH((\2), \1, \3);", src)
    cpp = d / "global.cpp"
    cpp.write_text('#include "cuda_blocks.h"\n' + src + MAIN)
    so = str(d / "global.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I",
                    os.path.join(HERE, "emulation"), "-I", CSRC,
                    "-I", "/usr/local/cuda/include", str(cpp), "-o", so], check=True)
    lib = C.CDLL(so)

    def run(cur, ref, rng, order):
        h, w = cur.shape
        dxdy, sad, why = (C.c_int * 2)(), C.c_ulonglong(), C.create_string_buffer(256)
        rc = lib.emulate(cur.ctypes.data_as(C.c_void_p), ref.ctypes.data_as(C.c_void_p), w, h, rng, order, dxdy,
                         C.byref(sad), why, C.c_size_t(256))
        return rc, why.value.decode(), (dxdy[0], dxdy[1], sad.value)

    def calls(pic, streams, capturing=False):
        h, w = pic.shape
        out = C.create_string_buffer(1 << 16)
        ptr = pic.ctypes.data_as(C.c_void_p)
        rc = lib.emulate_calls(ptr, ptr, w, h, (C.c_size_t * len(streams))(*streams), len(streams), int(capturing), out,
                               C.c_size_t(1 << 16))
        assert rc == 0, out.value
        return out.value.decode().split("\n")[:-1]

    run.calls = calls
    return run


# moved by (dx, dy): a best coarse vector at the range's lower corner leaves the refinement's first
# slots empty; 32 is the extended search; 0 the single frame SAD
@pytest.mark.parametrize("order", ["in order", "late warps"])
@pytest.mark.parametrize("rng,dx,dy", [(0, 0, 0), (1, -1, -1), (3, -3, -3), (3, 2, 1), (32, -32, 8)])
def test_stage_fold_waits_for_every_warp(search, oracle, rng, dx, dy, order):
    w, h = 80, 70  # 70 rows: two slabs at full resolution
    yy, xx = np.mgrid[0:h + 80, 0:w + 80]
    t = 128 + 60 * np.sin(xx / 7.3) + 50 * np.cos(yy / 5.1 + xx / 19)
    t = np.clip(np.rint(t), 0, 255).astype(np.uint8)
    cur = np.ascontiguousarray(t[40:40 + h, 40:40 + w])
    ref = np.ascontiguousarray(t[40 - dy:40 - dy + h, 40 - dx:40 - dx + w])
    c = np.full((h // 2, w // 2), 128, np.uint8)
    want = oracle.global_motion(make_params(w, h), (cur, c, c), (ref, c, c), rng)
    rc, why, got = search(cur, ref, rng, ["in order", "late warps"].index(order))
    assert rc == 0, why
    assert got == tuple(int(v) for v in want)


def test_calls_that_share_the_array_run_in_order(search):
    pic = np.zeros((16, 16), np.uint8)
    done = []  # (stream, event) of the last record
    first = True
    for line in search.calls(pic, [1, 2, 2, 3]):
        what, *v = line.split()
        if what == "record":
            done, first = [v[0], v[1]], True
        elif what == "wait":
            assert not done or v[1] == done[1]
            done = []
        else:  # a call's first launch comes after the wait for the last call's record
            assert not first or not done, line
            first = False
    assert done  # the last call left its record
    # a captured call takes no part: an event outside its capture would end the capture
    assert {line.split()[0] for line in search.calls(pic, [1, 2], capturing=True)} == {"launch"}
