"""How a call's core passes are planned: which seeds are refused, and which passes share a launch.

A seed is read by macroblock index, so a pass takes any seed of as many macroblocks, in the call or
from an earlier one alike. A seeded step runs as one launch while its passes' wavefront fronts
together stay within 8 macroblocks per SM, else as one launch per MV mode: the results on both
sides of the line are those of the passes one by one.
"""
import pytest

from libvc1_b200 import synth
from libvc1_b200.abi import MV_HPEL, MV_HPEL_BILINEAR, MV_MIXED, MV_QPEL, make_params

pytestmark = pytest.mark.gpu

MODES = (MV_HPEL, MV_HPEL_BILINEAR, MV_MIXED)


def _params(w, h):
    return make_params(w, h, search_range=16, local_search_range=16)


def _upload(ctx, w, h, first, seed):
    clip = synth.generate(w, h, 2, seed, global_px=4.0, n_objects=1, obj_min=16, obj_max=32)
    ctx.upload_frame(first, *clip.frame(0))
    ctx.upload_frame(first + 1, *clip.frame(1))


def test_a_seed_of_as_many_macroblocks_is_taken(ctx):
    wide, tall = _params(320, 160), _params(160, 320)
    _upload(ctx, 320, 160, 0, 5)
    _upload(ctx, 160, 320, 2, 6)
    first, second = (1, 0, MV_QPEL, 0, -1, 50), (3, 2, MV_MIXED, 1, 50, 51)
    ctx.core_passes(wide, [first])
    ctx.core_passes(tall, [second])  # the seed from an earlier call
    want = ctx.read_result(tall, 51)
    ctx.core_passes_multi([wide, tall], [(1, 0, MV_QPEL, 0, -1, 60), (3, 2, MV_MIXED, 1, 60, 61)])
    assert ctx.read_result(tall, 61).equal(want) == []


def test_refused_seeds(ctx):
    from libvc1_b200.api import Vc1cuError

    small, large = _params(96, 64), _params(160, 96)
    _upload(ctx, 96, 64, 0, 7)
    _upload(ctx, 160, 96, 2, 8)
    ctx.core_passes(small, [(1, 0, MV_QPEL, 0, -1, 70)])
    kept = ctx.read_result(small, 70)
    with pytest.raises(Vc1cuError) as e:  # a raster of another size, in the call and before it
        ctx.core_passes_multi([small, large], [(1, 0, MV_QPEL, 0, -1, 71), (3, 2, MV_QPEL, 0, 71, 72)])
    assert e.value.code == 1
    with pytest.raises(Vc1cuError) as e:
        ctx.core_passes(large, [(3, 2, MV_QPEL, 0, 70, 72)])
    assert e.value.code == 5
    with pytest.raises(Vc1cuError) as e:  # passes that seed each other
        ctx.core_passes(small, [(1, 0, MV_QPEL, 0, 74, 73), (1, 0, MV_QPEL, 0, 73, 74)])
    assert e.value.code == 1 and "cycle" in str(e.value)
    with pytest.raises(Vc1cuError) as e:
        ctx.core_passes(small, [(1, 0, MV_QPEL, 0, 73, 73)])
    assert e.value.code == 1
    # nothing of a refused call was launched
    assert ctx.read_result(small, 70).equal(kept) == []


def test_modes_in_one_launch_and_in_one_each(ctx):
    """320x336 holds 10 macroblocks in a wavefront step: three modes of 39 pictures stay within 8 per
    SM of a 148-SM device (1170 of 1184), of 40 they do not."""
    w, h = 320, 336
    p = _params(w, h)
    _upload(ctx, w, h, 0, 9)
    ctx.core_passes(p, [(1, 0, MV_QPEL, 0, -1, 1000)])
    want = []
    for j, m in enumerate(MODES):
        ctx.core_passes(p, [(1, 0, m, 0, 1000, 1001 + j)])
        want.append(ctx.read_result(p, 1001 + j))
    for n in (1, 39, 40):
        ctx.reset_counters()
        ctx.core_passes(p, [(1, 0, m, 0, 1000, 1010 + 3 * k + j) for k in range(n) for j, m in enumerate(MODES)])
        assert ctx.counters()["dispatches"] == (1 if n < 40 else 3), n
        for k in range(n):
            for j in range(3):
                assert ctx.read_result(p, 1010 + 3 * k + j).equal(want[j]) == [], (n, k, j)
