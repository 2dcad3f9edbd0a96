"""The UMH search and the staged refinement against the oracle where their parallel forms can go
wrong: ranges on both sides of every step change of the search (7/8 the lattice, 23/24 and 95/96
the rings and the cross, 31/32 the rescue's dense scan) and not divisible by the lattice's 8 or the
rescue's 4 (the far edges), pictures of one macroblock, with partial macroblocks and cropped
displays, and contents that tie every candidate (flat), match nowhere (unrelated noise: the
rescue) or match beyond the picture's edges."""
import numpy as np
import pytest

from libvc1_b200.abi import MV_HPEL_BILINEAR, MV_MIXED, MV_QPEL, make_params

pytestmark = pytest.mark.gpu

SIZES = [(16, 16, 0), (18, 34, 0), (50, 36, 3), (98, 66, 5)]


def _frames(kind, w, h, seed):
    rng = np.random.default_rng(seed)
    if kind == "flat":
        y = np.full((h, w), 70, np.uint8)
        pair = (y, y.copy())
    elif kind == "unrelated":
        pair = (rng.integers(0, 256, (h, w)).astype(np.uint8), rng.integers(0, 256, (h, w)).astype(np.uint8))
    else:  # smooth texture moved by more than a macroblock, so that matches reach over the edges
        yy, xx = np.mgrid[0:h + 64, 0:w + 64]
        t = 128 + 50 * np.sin(xx / 3.1) + 40 * np.cos(yy / 4.3) + rng.normal(0, 4, xx.shape)
        t = np.clip(np.rint(t), 0, 255).astype(np.uint8)
        pair = (t[20:20 + h, 37:37 + w].copy(), t[:h, 9:9 + w].copy())
    u = rng.integers(110, 146, (h // 2, w // 2)).astype(np.uint8)
    return [(y, u, u.copy()) for y in pair]


@pytest.mark.parametrize("kind", ["flat", "unrelated", "moved"])
@pytest.mark.parametrize("rng", [1, 2, 7, 8, 9, 23, 24, 31, 32, 33, 95, 96, 102])
def test_passes_match_oracle(ctx, oracle, rng, kind):
    for k, (w, h, crop) in enumerate(SIZES):
        cur, ref = _frames(kind, w, h, 10 * rng + k)
        kw = dict(display_width=w - crop, display_height=h - crop) if crop else {}
        p = make_params(w, h, search_range=rng, local_search_range=rng, pqindex=2 + rng % 17, rnd=k & 1, **kw)
        ctx.upload_frame(0, *ref)
        ctx.upload_frame(1, *cur)
        for mode in (MV_QPEL, MV_HPEL_BILINEAR):
            got = ctx.analyze_p_core(p, 1, 0, mode, False)
            assert got.equal(oracle.analyze_p_core(p, cur, ref, mode, False)) == [], (w, h, mode)
        seed = oracle.analyze_p_core(p, cur, ref, MV_QPEL, False)
        got = ctx.analyze_p_core(p, 1, 0, MV_MIXED, True, seed=seed.mvs, seed_distant=seed)
        assert got.equal(oracle.analyze_p_core(p, cur, ref, MV_MIXED, True, seed=seed.mvs, seed_distant=seed)) == [], (w, h)


def test_largest_local_range(ctx, oracle):
    """Range 190, the largest local range, and the refusal above it."""
    from libvc1_b200.api import Vc1cuError

    cur, ref = _frames("moved", 50, 36, 3)
    ctx.upload_frame(0, *ref)
    ctx.upload_frame(1, *cur)
    p = make_params(50, 36, search_range=190, local_search_range=190)
    assert ctx.analyze_p_core(p, 1, 0, MV_QPEL, False).equal(oracle.analyze_p_core(p, cur, ref, MV_QPEL, False)) == []
    with pytest.raises(Vc1cuError) as e:
        ctx.analyze_p_core(make_params(50, 36, search_range=191, local_search_range=191), 1, 0, MV_QPEL, False)
    assert e.value.code == 6


@pytest.mark.parametrize("rng", [32, 64])
@pytest.mark.parametrize("n", [1, 64, 119])
def test_launch_shapes(ctx, oracle, rng, n):
    """n equal pairs in one call: the fronts of few, of more and of twice as many macroblocks as four
    warps per SM hold, each with its own blocks per SM or warps per block."""
    w, h = 320, 336
    cur, ref = _frames("moved", w, h, rng)
    p = make_params(w, h, search_range=rng, local_search_range=rng)
    ctx.upload_frame(0, *ref)
    ctx.upload_frame(1, *cur)
    ctx.core_passes(p, [(1, 0, MV_QPEL, 0, -1, k) for k in range(n)])
    ctx.core_passes(p, [(1, 0, MV_MIXED, 1, k, n + k) for k in range(n)])
    want = oracle.analyze_p_core(p, cur, ref, MV_QPEL, False)
    mixed = oracle.analyze_p_core(p, cur, ref, MV_MIXED, True, seed=want.mvs, seed_distant=want)
    for k in range(n):
        assert ctx.read_result(p, k).equal(want) == [], k
        assert ctx.read_result(p, n + k).equal(mixed) == [], k
