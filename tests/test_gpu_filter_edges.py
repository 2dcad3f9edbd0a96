"""The deblocking stages against the oracle's raster-order filters at the sizes where their line
groups end: pictures of one macroblock, widths and heights that leave two columns or rows of a
group (its deciding third line missing), odd chroma sizes, partial macroblocks, and metadata that
filters every border, only coded patterns, or nothing."""
import numpy as np
import pytest

from libvc1_b200.abi import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(16, 16), (18, 18), (20, 22), (26, 30), (34, 50), (46, 36), (130, 70)])
@pytest.mark.parametrize("meta_kind", ["dense", "one_vector", "uncoded"])
def test_loop_filters_match_oracle(ctx, oracle, size, meta_kind):
    from lf_cases import blocky_frame, metadata

    w, h = size
    for pq in (3, 12, 31):
        p = make_params(w, h, pqindex=pq)
        fr = blocky_frame(w, h, w + h + pq)
        bmv, cbp, tt, intra = metadata(w, h, w * pq, meta_kind == "dense")
        if meta_kind != "dense":
            bmv[:] = 0
            intra[:] = 0
        if meta_kind == "uncoded":
            cbp[:] = 0
        ctx.upload_frame(0, *fr)
        ctx.loop_filter(p, 0, bmv, cbp, tt, intra)
        want = oracle.loop_filter(p, fr, bmv, cbp, tt, intra)
        assert all(np.array_equal(a, b) for a, b in zip(ctx.download_frame(0, w, h), want)), pq
        ctx.upload_frame(0, *fr)
        ctx.loop_filter(p, 0)
        assert all(np.array_equal(a, b) for a, b in zip(ctx.download_frame(0, w, h), oracle.loop_filter(p, fr))), pq
