"""The transform RD, the DQUANT search and the intra reconstruction against golden results
(tests/golden/trd_kat.npz) at the edges of their parallel forms: rasters of one macroblock, with
partial macroblocks and cropped displays, every trellis beam, coding sets with and without
Escape-3 headers, pictures that match, differ and share nothing. The fixture was written by the
build whose transform RD, DQUANT search and intra reconstruction had been compared with the
reference's own functions bit for bit (tests/test_gpu_transform_rd.py, test_gpu_dquant.py and
test_gpu_intra.py, which run where the reference's checker library is built)."""
import os

import numpy as np
import pytest

from libvc1_b200.abi import TDECISION_DTYPE, make_params, make_trd_cfg, mbs_of

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "trd_kat.npz")

# (w, h, crop, pq, parameters, transform RD configuration, content)
CASES = [
    (16, 16, 0, 3, {}, dict(trellis=1), "natural"),
    (18, 34, 0, 12, dict(nonuniform=1), dict(trellis=2, coding_set=3), "dark_detail"),
    (50, 36, 3, 6, dict(halfqp=1), dict(trellis=1, aq_strength=2.5), "adjacency"),
    (64, 48, 0, 1, {}, dict(trellis=2, hrd_enabled=1), "unrelated"),
    (66, 50, 5, 8, {}, dict(trellis=0, coding_set=5), "bright_on_dark"),
    (64, 48, 0, 20, dict(nonuniform=1), dict(trellis=1, extended_transform_signaling=0), "natural"),
    (48, 64, 0, 4, {}, dict(trellis=1, use_vlc=0), "coarser"),
    (64, 48, 0, 9, {}, dict(trellis=1, variable_transforms=0, coding_set=7), "natural"),
    (64, 48, 1, 14, {}, dict(trellis=2, frame_type=4, adaptive_quality=0), "dark_detail"),
]


def results(ctx, i):
    """Every output of case i, as flat arrays."""
    import torch
    from dq_cases import frames

    w, h, crop, pq, par, cfg, kind = CASES[i]
    kw = dict(display_width=w - crop, display_height=h - crop) if crop else {}
    p = make_params(w, h, pqindex=pq, **par, **kw)
    mbw, mbh = mbs_of(p)
    src, pred = frames("natural" if kind == "unrelated" else kind, w, h, 40 + i)
    rng = np.random.default_rng(70 + i)
    if kind == "unrelated":
        pred = tuple(rng.integers(0, 256, a.shape).astype(np.uint8) for a in pred)
    c = make_trd_cfg(**cfg)
    ctx.upload_frame(0, *src)
    ctx.upload_frame(1, *pred)
    base = np.clip(pq + rng.integers(-1, 3, mbw * mbh), 1, 31).astype(np.uint8)
    out = {}
    for name, (d, *rest) in (("trd", ctx.choose_transform(p, c, 0, 1, mquant=base if i % 2 else None)),
                             ("dq", ctx.choose_dquant(p, c, 0, 1, base))):
        for f in TDECISION_DTYPE.names:
            if f != "reserved":
                out[f"{name}.{f}"] = np.ascontiguousarray(d[f])
        for k, a in enumerate(rest):
            out[f"{name}.{k}"] = a
    planes = [torch.zeros((16 * mbh >> s, 16 * mbw >> s), dtype=torch.int32, device="cuda") for s in (0, 1, 1)]
    torch.cuda.synchronize()
    ctx.reconstruct_intra(p, 0, *[t.data_ptr() for t in planes], overlap=i % 2, mquant=base,
                          derived=(base != pq).astype(np.uint8), cfg=c)
    ctx.synchronize()
    for k, t in enumerate(planes):
        out[f"intra.{k}"] = t.cpu().numpy().astype(np.int16)
    return out


@pytest.mark.parametrize("i", range(len(CASES)))
def test_matches_golden(ctx, i):
    g = np.load(GOLDEN)
    for name, a in results(ctx, i).items():
        want = g[f"c{i}.{name}"]
        if a.dtype == np.float64:
            a, want = a.view(np.uint64), want.view(np.uint64)
        assert np.array_equal(a, want), name
