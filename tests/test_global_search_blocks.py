"""The global translation search's kernels run on the host, thread by thread, under chosen orders.

A stage's last block to finish folds its costs and rewrites the candidate list that every block of
the stage has read. So no warp may still have its candidate to read once its block counts as
finished, however late that warp runs: the order "late warps" lets the first warp of each block run
ahead and holds the rest of a finished block back until nothing else can advance. The kernels'
source itself is compiled (emulation/cuda_blocks.h); the results are the oracle's.
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
