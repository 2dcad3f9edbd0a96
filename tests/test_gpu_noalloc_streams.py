"""vc1cu_global_motion_noalloc from several streams and threads: its calls share one array per device,
so that each must wait for the work of the call before it. Pictures of different sizes, every
result the oracle's; and a captured call replayed."""
import threading

import numpy as np
import pytest

from libvc1_b200 import synth
from libvc1_b200.abi import make_params

pytestmark = pytest.mark.gpu

CASES = [(1280, 720, 32, 8), (64, 48, 8, 16), (322, 242, 12, 1), (352, 288, 0, 3)]  # size, range, pictures


@pytest.fixture(scope="module")
def pictures(oracle):
    torch = pytest.importorskip("torch")
    out = []
    for w, h, rng, n in CASES:
        clip = synth.generate(w, h, 2, w, global_px=6.0, n_objects=1, obj_min=8, obj_max=16)
        cur, ref = clip.frame(1), clip.frame(0)
        want = tuple(int(v) for v in oracle.global_motion(make_params(w, h), cur, ref, rng))
        dev = [torch.from_numpy(np.ascontiguousarray(f[0])).cuda() for f in (cur, ref)]
        out.append((w, h, rng, n, dev, want))
    torch.cuda.synchronize()
    return out


def _call(torch, pic, stream):
    from libvc1_b200.api import global_motion_noalloc

    w, h, rng, n, (cur, ref), _ = pic
    dxdy = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    sad = torch.empty(n, dtype=torch.int64, device="cuda")
    global_motion_noalloc([cur.data_ptr()] * n, [ref.data_ptr()] * n, w, w, h, rng, dxdy.data_ptr(), sad.data_ptr(),
                          stream.cuda_stream)
    return dxdy, sad


def _check(pic, got):
    dxdy, sad = got[0].cpu().numpy().reshape(-1, 2), got[1].cpu().numpy()
    assert [(int(d[0]), int(d[1]), int(s)) for d, s in zip(dxdy, sad)] == [pic[5]] * pic[3]


def test_streams(pictures):
    import torch

    streams = [torch.cuda.Stream() for _ in range(3)]
    runs = [(pictures[k % 4], streams[k % 3]) for k in range(24)]
    got = [_call(torch, pic, s) for pic, s in runs]
    torch.cuda.synchronize()
    for (pic, _), g in zip(runs, got):
        _check(pic, g)


def test_threads(pictures):
    import torch

    got = [[] for _ in range(4)]

    def work(k):
        s = torch.cuda.Stream()
        for _ in range(8):
            got[k].append(_call(torch, pictures[k], s))
        s.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        assert len(got[k]) == 8
        for g in got[k]:
            _check(pictures[k], g)


def test_captured_call(pictures):
    import torch

    pic = pictures[2]
    s = torch.cuda.Stream()
    _call(torch, pic, s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        got = _call(torch, pic, s)
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        _check(pic, got)
