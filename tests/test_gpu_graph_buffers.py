"""Graph replays after calls that outgrow the context's workspaces.

A graph's nodes hold the addresses of the context's buffers (search states, pass and B-picture
descriptors, prediction planes, signature indexes). A later, larger call replaces them; the replay
must still write what the recorded calls wrote. A slot that has had another size since is refused.
"""
import numpy as np
import pytest

from libvc1_b200 import synth
from libvc1_b200.abi import MV_MIXED, MV_QPEL, make_params

pytestmark = pytest.mark.gpu


@pytest.fixture()
def own():
    """A context of the test's own: its workspaces start empty, so that the first calls size them."""
    from libvc1_b200.api import CudaComputeContext

    c, err = CudaComputeContext.create(0)
    assert c is not None, err
    yield c
    c.close()


def _upload(c, w, h, seed, first):
    clip = synth.generate(w, h, 3, seed, global_px=5.0, n_objects=1, obj_min=16, obj_max=32)
    for t in range(3):
        c.upload_frame(first + t, *clip.frame(t))


def _calls(c, p):
    """A P pass chain and a B picture over the frames 0, 1, 2 (past, current, future)."""
    c.core_passes(p, [(2, 0, MV_QPEL, 0, -1, 0), (2, 0, MV_MIXED, 1, 0, 1)])
    c.core_passes(p, [(1, 0, MV_QPEL, 0, -1, 2), (1, 2, MV_QPEL, 0, -1, 3)])
    c.b_decide(p, [(1, 0, 2, 2, 3, 1, 1, 2, MV_QPEL, 0)])


def _results(c, p):
    return [c.read_result(p, k) for k in range(4)], c.read_bresult(p, 0)


@pytest.mark.parametrize("search,local", [(16, 16), (64, 16)])
def test_replay_after_larger_calls(own, search, local):
    c = own
    small = make_params(96, 64, search_range=search, local_search_range=local)
    _upload(c, 96, 64, 7, 0)
    _calls(c, small)
    want, want_b = _results(c, small)
    c.graph_begin()
    _calls(c, small)
    g = c.graph_end()
    try:
        # more passes, B pictures and references than the capture had, over a larger raster
        large = make_params(320, 240, search_range=search, local_search_range=local)
        for k in range(3):
            _upload(c, 320, 240, 20 + k, 100 + 3 * k)
        c.core_passes(large, [(100 + 3 * k + (d + 1), 100 + 3 * k, MV_QPEL, 0, -1, 100 + 2 * k + d)
                              for k in range(3) for d in range(2)])
        c.core_passes(large, [(101 + 3 * k, 102 + 3 * k, MV_QPEL, 0, -1, 200 + k) for k in range(3)])
        c.b_decide(large, [(101 + 3 * k, 100 + 3 * k, 102 + 3 * k, 100 + 2 * k, 200 + k, 101 + 2 * k, 1, 2, MV_QPEL,
                            100 + k)
                           for k in range(3)])
        c.synchronize()
        for _ in range(2):
            c.graph_launch(g)
            got, got_b = _results(c, small)
            assert all(a.equal(b) == [] for a, b in zip(got, want))
            assert got_b.equal(want_b) == []
    finally:
        c.graph_destroy(g)


@pytest.mark.parametrize("slot", ["frame", "result"])
def test_replay_refused_after_a_slot_changed_size(own, slot):
    from libvc1_b200.api import Vc1cuError

    c = own
    p = make_params(96, 64, search_range=8, local_search_range=8)
    _upload(c, 96, 64, 3, 0)
    passes = [(2, 0, MV_QPEL, 0, -1, 0)]
    c.core_passes(p, passes)
    want = c.read_result(p, 0)
    c.graph_begin()
    c.core_passes(p, passes)
    g = c.graph_end()
    try:
        other = make_params(128, 80, search_range=8, local_search_range=8)
        _upload(c, 128, 80, 4, 0 if slot == "frame" else 10)
        if slot == "result":
            c.core_passes(other, [(12, 10, MV_QPEL, 0, -1, 0)])
        with pytest.raises(Vc1cuError) as e:
            c.graph_launch(g)
        assert e.value.code == 5 and "size" in str(e.value)
        # the context goes on working
        _upload(c, 96, 64, 3, 20)
        c.core_passes(p, [(22, 20, MV_QPEL, 0, -1, 5)])
        assert c.read_result(p, 5).equal(want) == []
    finally:
        c.graph_destroy(g)


def test_replay_keeps_the_recorded_host_arrays(own):
    """The host arrays of captured calls may change or go after the capture."""
    torch = pytest.importorskip("torch")
    c = own
    w, h, mbs = 96, 64, 24
    p = make_params(w, h, search_range=8, local_search_range=8, pqindex=4)
    _upload(c, w, h, 5, 0)
    lv = torch.empty((4, mbs, 6, 64), dtype=torch.int16, device="cuda")
    c.forward_quant_device(p, 1, 0, 15, 0, lv.data_ptr())
    signed = [torch.arange(n, dtype=torch.int32, device="cuda") % 255 for n in (w * h, w * h // 4, w * h // 4)]
    torch.cuda.synchronize()
    rng = np.random.default_rng(1)
    types = rng.integers(1, 5, (mbs, 6)).astype(np.uint8)
    mask = rng.integers(0, 2, mbs).astype(np.uint8)

    def calls():
        c.reconstruct(p, 0, lv.data_ptr(), 15, types, 3)
        c.store_signed(p, *[s.data_ptr() for s in signed], 0, 3, mask)

    calls()
    want = c.download_frame(3, w, h)
    c.graph_begin()
    calls()
    g = c.graph_end()
    try:
        types[:] = 5 - types
        mask[:] = 1 - mask
        calls()
        assert any(not np.array_equal(a, b) for a, b in zip(c.download_frame(3, w, h), want))
        c.graph_launch(g)
        for a, b in zip(c.download_frame(3, w, h), want):
            assert np.array_equal(a, b)
    finally:
        c.graph_destroy(g)
