"""The whole-frame translation search against the oracle at the sizes and contents where its
parallel folds can go wrong: every range class (none, the plain search's three coarse steps, the
extended search's 32), pictures narrower than a 16-pixel chunk and with ragged last chunks,
planes at unaligned addresses with odd pitches, and contents whose costs tie (flat and periodic
pictures), where the result is decided by the visit order alone."""
import numpy as np
import pytest

from libvc1_b200.abi import make_params

pytestmark = pytest.mark.gpu


def _pictures(kind, w, h, seed):
    rng = np.random.default_rng(seed)
    if kind == "flat":
        a = np.full((h, w), 90, np.uint8)
        return a, a.copy()
    if kind == "periodic":
        yy, xx = np.mgrid[0:h, 0:w]
        a = (100 + 60 * ((xx // 4 + yy // 4) & 1)).astype(np.uint8)
        return a, np.roll(a, (3, 5), (0, 1))
    a = rng.integers(0, 256, (h, w)).astype(np.uint8)
    return a, np.roll(a, (-6, 9), (0, 1))


@pytest.mark.parametrize("rng", [0, 1, 2, 3, 4, 7, 8, 30, 31, 32])
@pytest.mark.parametrize("kind", ["flat", "periodic", "noise"])
@pytest.mark.parametrize("size", [(14, 10), (16, 16), (50, 34), (130, 98), (338, 70)])
def test_global_search_matches_oracle(oracle, size, kind, rng):
    torch = pytest.importorskip("torch")
    from libvc1_b200.api import global_motion_noalloc

    w, h = size
    cur, ref = _pictures(kind, w, h, w + rng)
    u = np.zeros((h // 2, w // 2), np.uint8)
    want = oracle.global_motion(make_params(w, h), (cur, u, u), (ref, u, u), rng)
    pitch, off = w + 3, 1  # rows and planes at every alignment
    planes = []
    for pl in (cur, ref):
        host = np.zeros(off + h * pitch, np.uint8)
        host[off:].reshape(h, pitch)[:, :w] = pl
        planes.append(torch.from_numpy(host).cuda())
    dxdy = torch.zeros(4, dtype=torch.int32, device="cuda")
    sad = torch.zeros(2, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream()
    p = [t.data_ptr() + off for t in planes]
    global_motion_noalloc([p[0], p[1]], [p[1], p[1]], pitch, w, h, rng, dxdy.data_ptr(), sad.data_ptr(), s.cuda_stream)
    s.synchronize()
    got = dxdy.cpu().numpy(), sad.cpu().numpy()
    assert (int(got[0][0]), int(got[0][1]), int(got[1][0])) == tuple(int(x) for x in want)
    assert (got[0][2], got[0][3], got[1][1]) == (0, 0, 0)  # a picture against itself
