"""The work that programs built on this library have it do, as cases to be timed.

Every case is one pass through the public entry points of libvc1_b200.api on seeded synthetic
pictures (the library's own clip generator). The kinds and what each stands for in real use:

- score: one batch of motion candidates of a block through the motion-compute backend interface
  (score_motion_batch); the smallest call a host encoder makes.
- p_core: a host encoder that runs one analysis pass at a time: the picture is uploaded, the
  unseeded quarter-pel pass is analysed, its vectors go back to the device as the seed of a
  Mixed-MV pass with P-intra. CIF and smaller sizes, where launches and latency count.
- p_picture: an encoder's whole decision on one P picture: the scene-cut score, then
  analyze_p_picture with the default presets (five passes, motion bits, sampled transform RD, fade
  estimate), and the analysis read back.
- b_picture: one B picture's analysis against host anchor vectors, synchronous.
- gop: a GOP of IBBP pictures resident on the device, every picture in one batch per stage: the
  benchmark's throughput form (seed, mode and final passes, prediction, the four transform sizes'
  levels, B decisions, results read back).
- clips: one frame step of clips of uneven sizes in one launch (five chained passes per clip).
- longrange: unseeded passes of pictures with camera pans at the extended motion range.
- transform: the default presets' transform RD of a predicted picture, without or with the DQUANT
  search.
- recon: the reconstruction of a coded P picture: levels of the four transform sizes, the inverse
  transforms, the in-loop filter.
- intra: an I picture: its overlap plan, the signed reconstruction, overlap smoothing, the store
  and the in-loop filter.
- learned: picture pairs through the learned proposals (features, network, learned pass with the
  plain fallback).
- train: one batch's loss and gradients of the proposal network (forward and backward).

Sizes run from 96x64 to 1920x1080, even and odd macroblock counts, cropped displays among them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from libvc1_b200 import learned, synth
from libvc1_b200.abi import (MV_HPEL, MV_HPEL_BILINEAR, MV_MIXED, MV_QPEL, TDECISION_DTYPE, make_ppic_cfg, make_params,
                             make_trd_cfg, mbs_of)
from libvc1_b200.api import CudaComputeContext, LearnedProposals

MODES = (MV_HPEL, MV_HPEL_BILINEAR, MV_MIXED)


def listed():
    return [
        # the backend interface's smallest call: one 16x16 block's candidates in a CIF picture
        dict(name="score_16x16", kind="score", w=352, h=288, block=16, n=64, satd=False, bilinear=False, stride=1),
        # one picture at a time at CIF: the plain CIF configuration (UMH, range 32, QP 8)
        dict(name="p_core_cif", kind="p_core", w=352, h=288, crop=0, range=32, local=32, diamond=False, fast=False, pq=8),
        # a P picture's whole decision at 1080p with the default presets
        dict(name="p_picture_1080p", kind="p_picture", w=1920, h=1080, crop=0, range=64, local=64, pq=6, nonuniform=True),
        # a B picture at 720p, half-way between its anchors
        dict(name="b_picture_720p", kind="b_picture", w=1280, h=720, crop=0, range=64, local=64, pq=8, num=1, den=2,
             bilinear=False),
        # the benchmark's throughput form: one 1080p GOP 12 IBBP (4 P and 7 B pictures)
        dict(name="gop_1080p", kind="gop", w=1920, h=1080, frames=12, range=64, pq=6),
        # one frame step of the batched clips: three sizes and two odd ones
        dict(name="clips_uneven", kind="clips", clips=6, big=1920, range=32, pq=8, odd=77),
        # extended motion range: two 1080p pictures of pans of up to 200 pixels
        dict(name="longrange_1080p", kind="longrange", w=1920, h=1080, pictures=2, range=1024, local=32, pan=200, pq=6),
        # the default presets' transform RD of a 1080p picture (trellis, perceptual scale)
        dict(name="transform_rd_1080p", kind="transform", w=1920, h=1080, crop=0, pq=6, nonuniform=False, trellis=1,
             dquant=False),
        # the reconstruction of a 1080p picture in a cropped raster
        dict(name="recon_p_1080p", kind="recon", w=1920, h=1080, crop=0, pq=8, nonuniform=True, coeffs=False),
        # an I picture at an odd display size
        dict(name="intra_odd", kind="intra", w=1278, h=722, crop=5, pq=8, nonuniform=False, trellis=1),
        # the learned form on 1080p pairs
        dict(name="learned_1080p", kind="learned", w=1920, h=1080, pairs=4, range=128, local=32, pan=128),
        # a training batch of the proposal network
        dict(name="train_1080p", kind="train", w=1920, h=1080, pairs=4, range=128, local=32, pan=128),
    ]


def _size(rng, lo, hi):
    """An even size in lo..hi, spread over its logarithm."""
    return 2 * max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2)))


def draw(rng):
    kind = rng.choice(["score", "p_core", "p_picture", "b_picture", "gop", "clips", "longrange", "transform", "recon",
                       "intra", "learned", "train"])
    w, h = _size(rng, 96, 1920), _size(rng, 64, 1080)
    crop = rng.choice([0, 0, 1, 3, 5])
    pq = rng.randint(2, 20)
    if kind == "score":
        return dict(kind=kind, w=w, h=h, block=rng.choice([8, 16]), n=int(math.exp(rng.uniform(math.log(8), math.log(4096)))),
                    satd=rng.random() < 0.5, bilinear=rng.random() < 0.3, stride=1)
    if kind == "p_core":
        r = rng.choice([8, 16, 32, 48, 64])
        return dict(kind=kind, w=min(w, 1280), h=min(h, 720), crop=crop, range=r, local=rng.choice([r, min(r, 16)]),
                    diamond=rng.random() < 0.3, fast=rng.random() < 0.3, pq=pq)
    if kind == "p_picture":
        r = rng.choice([16, 32, 64])
        return dict(kind=kind, w=w, h=h, crop=crop, range=r, local=r, pq=pq, nonuniform=rng.random() < 0.5)
    if kind == "b_picture":
        num, den = rng.choice([(1, 2), (1, 3), (2, 3)])
        r = rng.choice([16, 32, 64])
        return dict(kind=kind, w=w, h=h, crop=crop, range=r, local=r, pq=pq, num=num, den=den, bilinear=rng.random() < 0.5)
    if kind == "gop":
        return dict(kind=kind, w=w, h=h, frames=rng.randint(4, 12), range=rng.choice([16, 32, 64]), pq=pq)
    if kind == "clips":
        return dict(kind=kind, clips=rng.randint(2, 6), big=rng.choice([640, 1280, 1920]), range=rng.choice([16, 32]), pq=pq,
                    odd=rng.randint(1, 1000))
    if kind == "longrange":
        return dict(kind=kind, w=max(w, 320), h=max(h, 240), pictures=rng.randint(1, 2), range=rng.choice([128, 512, 1024]),
                    local=32, pan=rng.choice([60, 120, 200]), pq=pq)
    if kind == "transform":
        return dict(kind=kind, w=w, h=h, crop=crop, pq=pq, nonuniform=rng.random() < 0.5, trellis=rng.randint(0, 2),
                    dquant=rng.random() < 0.5)
    if kind == "recon":
        return dict(kind=kind, w=w, h=h, crop=crop, pq=pq, nonuniform=rng.random() < 0.5, coeffs=rng.random() < 0.5)
    if kind == "intra":
        return dict(kind=kind, w=w, h=h, crop=crop, pq=min(pq, 12), nonuniform=rng.random() < 0.5, trellis=rng.randint(0, 1))
    return dict(kind=kind, w=max(w, 320), h=max(h, 240), pairs=rng.randint(1, 4), range=rng.choice([64, 128]), local=32,
                pan=rng.choice([32, 64, 128]))


# ---- inputs ---------------------------------------------------------------------------------

def _params(case, **kw):
    w, h = case["w"], case["h"]
    crop = case.get("crop", 0)
    if crop:
        kw.update(display_width=w - crop, display_height=h - crop)
    r = case.get("range", 32)
    return make_params(w, h, search_range=r, local_search_range=case.get("local", r), pqindex=case.get("pq", 6),
                       nonuniform=int(case.get("nonuniform", False)), me_algorithm=int(case.get("diamond", False)),
                       fast_subpel=int(case.get("fast", False)), **kw)


def _context():
    ctx, err = CudaComputeContext.create(torch.cuda.current_device())
    if ctx is None:
        raise RuntimeError(err)
    return ctx


def _clip(ctx, w, h, frames, seed, first_id=0, pan=6.75, pan_y=None, objects=8, vel=8.0, zoom=1.002):
    """Frames 0.. of a seeded clip in frame slots first_id.."""
    side = max(8, min(32, min(w, h) // 4))
    cfg = synth.make_cfg(w, h, frames, seed, global_px=pan, global_py=pan_y, n_objects=objects, obj_min=side,
                         obj_max=3 * side, obj_vel=vel, zoom=zoom, sigma=2.0)
    ctx.synth_frames(cfg, 0, frames, first_id)


def _predicted(ctx, p, cur, ref, pred):
    """Frame slot `pred` = the Mixed-MV prediction of cur from ref (as an encoder has it before the
    transform); result slots 900 and 901."""
    ctx.core_passes(p, [(cur, ref, MV_QPEL, 0, -1, 900)])
    ctx.core_passes(p, [(cur, ref, MV_MIXED, 1, 900, 901)])
    ctx.motion_compensate(p, ref, 901, MV_MIXED, pred)


def _loop_filter_metadata(rng, p, types, bmv):
    """The coded-block metadata of a P picture with the given transform types: subblock patterns,
    filter kinds and a few intra blocks."""
    mbs = types.shape[0]
    skip = rng.integers(0, 16, types.shape)
    two = skip & 3
    pat = np.select([types == 1, types == 4, types == 2],
                    [np.full_like(skip, 15), ~skip & 15, ~((two & 2) * 6 + (two & 1) * 3) & 15], ~(two * 5) & 15)
    tt = np.array([0, 0, 3, 6, 7])[types]
    intra = (rng.random(mbs) < 0.05) * rng.integers(1, 64, mbs)
    return bmv, pat.astype(np.uint8), tt.astype(np.uint8), intra.astype(np.uint8)


def _clip_sizes(case):
    big = case["big"]
    sizes = [(640, 360, 0), (1280, 720, 0), (1920, 1080, 0)]
    out = [s for s in sizes if s[0] <= big]
    rng = np.random.default_rng(case["odd"])
    while len(out) < case["clips"]:
        dw, dh = int(rng.integers(161, 640)) * 2 + 1, int(rng.integers(121, 360)) * 2 + 1
        out.append((dw + 1, dh + 1, 1))
    return out[:case["clips"]]


def _learned_inputs(case, seed):
    """The pairs in frame slots 2k (current) and 2k + 1 (reference), and the network."""
    ctx = _context()
    w, h, n = case["w"], case["h"], case["pairs"]
    for k in range(n):
        cfg = synth.make_cfg(w, h, 2, 1000 * seed + k, global_px=float(case["pan"]), n_objects=8, obj_min=24, obj_max=96,
                             obj_vel=8.0, sigma=1.0 + k % 4)
        ctx.synth_frames(cfg, 1, 1, 2 * k)
        ctx.synth_frames(cfg, 0, 1, 2 * k + 1)
    net = LearnedProposals(ctx, w, h, case["range"], n, max_batch=n, seed=1)
    net.set_params(np.load(learned.WEIGHTS))
    p = _params(case)
    state = dict(case=case, ctx=ctx, net=net, p=p)
    if case["kind"] == "train":
        for k in range(n):
            net.prepare(2 * k, 2 * k + 1, k)
        ctx.core_passes(p, [(2 * k, 2 * k + 1, MV_QPEL, 0, -1, k) for k in range(n)])
        for k in range(n):
            net.set_labels(k, k)
    ctx.synchronize()
    return state


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("learned", "train"):
        return _learned_inputs(case, seed)
    s = dict(case=case, ctx=_context())
    ctx = s["ctx"]
    if kind == "score":
        clip = synth.generate(case["w"], case["h"], 2, seed, n_objects=4, obj_min=16, obj_max=32)
        b = case["block"]
        step = 2 if case["bilinear"] else 1
        s["cur"], s["ref"] = clip.y[1].copy(), clip.y[0].copy()
        s["x0"] = int(rng.integers(0, (case["w"] - b) // b + 1)) * b
        s["y0"] = int(rng.integers(0, (case["h"] - b) // b + 1)) * b
        s["cand"] = (rng.integers(-64, 65, (case["n"], 2)) * step).astype(np.int32)
        return s
    if kind == "clips":
        s["params"], s["passes"] = [], []
        for k, (w, h, crop) in enumerate(_clip_sizes(case)):
            _clip(ctx, w, h, 2, 100 * seed + k, 2 * k, pan=16.0, objects=4, vel=3.0, zoom=1.0)
            kw = dict(display_width=w - crop, display_height=h - crop) if crop else {}
            p = make_params(w, h, search_range=case["range"], local_search_range=case["range"], pqindex=case["pq"], **kw)
            s["params"] += [p] * 5
            cur, ref, base = 2 * k + 1, 2 * k, 5 * k
            s["passes"] += [(cur, ref, MV_QPEL, 0, -1, base)]
            s["passes"] += [(cur, ref, m, 0, base, base + 1 + j) for j, m in enumerate(MODES)]
            s["passes"] += [(cur, ref, MV_MIXED, 1, base + 3, base + 4)]
        ctx.synchronize()
        return s
    w, h = case["w"], case["h"]
    p = s["p"] = _params(case)
    mbw, mbh = mbs_of(p)
    mbs = mbw * mbh
    if kind == "p_core":
        clip = synth.generate(w, h, 2, seed, n_objects=4, obj_min=16, obj_max=32)
        ctx.upload_frame(0, *clip.frame(0))
        s["cur"] = tuple(a.copy() for a in clip.frame(1))
    elif kind == "p_picture":
        _clip(ctx, w, h, 2, seed)
        s["cfg"] = make_ppic_cfg()
    elif kind == "b_picture":
        _clip(ctx, w, h, 4, seed)
        ctx.core_passes(p, [(3, 0, MV_QPEL, 0, -1, 0)])
        ctx.core_passes(p, [(3, 0, MV_MIXED, 1, 0, 1)])
        a = ctx.read_result(p, 1)
        s["anchor"] = (a.mvs, a.use_4mv)
    elif kind == "gop":
        n = case["frames"]
        _clip(ctx, w, h, n, seed)
        s["pics"], s["bpics"], prev = [], [], 0
        while prev + 1 < n:
            nxt = min(prev + 3, n - 1)
            s["pics"].append((nxt, prev))
            s["bpics"] += [(j, prev, nxt, j - prev, nxt - prev, len(s["pics"]) - 1) for j in range(prev + 1, nxt)]
            prev = nxt
        s["levels"] = torch.empty((len(s["pics"]), 4, mbs, 6, 64), dtype=torch.int16, device="cuda")
    elif kind == "longrange":
        for k in range(case["pictures"]):
            _clip(ctx, w, h, 2, 100 * seed + k, 2 * k, pan=float(case["pan"]), pan_y=0.3 * case["pan"], objects=4)
    elif kind == "transform":
        _clip(ctx, w, h, 2, seed)
        _predicted(ctx, p, 1, 0, 2)
        s["cfg"] = make_trd_cfg(trellis=case["trellis"])
        base = case["pq"] + (rng.random(mbs) < 0.3) * rng.integers(-1, 3, mbs)
        s["base"] = np.clip(base, 1, 31).astype(np.uint8)
    elif kind == "recon":
        _clip(ctx, w, h, 2, seed)
        _predicted(ctx, p, 1, 0, 2)
        s["types"] = np.repeat(ctx.fast_transform_types(p, 1, 2)[:, None], 6, axis=1).copy()
        s["meta"] = _loop_filter_metadata(rng, p, s["types"].astype(np.int64), ctx.read_result(p, 901).block_mvs)
        s["levels"] = torch.empty((4, mbs, 6, 64), dtype=torch.int16, device="cuda")
        s["coeffs"] = torch.empty((4, mbs, 6, 64), dtype=torch.float64, device="cuda") if case["coeffs"] else None
    elif kind == "intra":
        _clip(ctx, w, h, 1, seed)
        s["cfg"] = make_trd_cfg(trellis=case["trellis"])
        s["planes"] = [torch.empty((16 * mbh >> c, 16 * mbw >> c), dtype=torch.int32, device="cuda") for c in (0, 1, 1)]
    ctx.synchronize()
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------------------

def _analysis(a):
    """The arrays and totals of an Analysis or BAnalysis."""
    out = {n: getattr(a, n) for n in a.ARRAYS}
    keys = sorted(a.totals)
    out["counts"] = np.array([a.totals[k] for k in keys if not isinstance(a.totals[k], float)], np.int64)
    out["means"] = np.array([a.totals[k] for k in keys if isinstance(a.totals[k], float)])
    return out


def _analyses(s, key, results):
    """Several analyses, field by field one after another, in buffers that the state keeps."""
    parts = [_analysis(a) for a in results]
    if key not in s:
        s[key] = {n: np.empty((sum(len(q[n]) for q in parts),) + v.shape[1:], v.dtype) for n, v in parts[0].items()}
    for n, dst in s[key].items():
        np.concatenate([q[n] for q in parts], out=dst)
    return s[key]


def _score(s):
    c = s["case"]
    ok, costs, err = s["ctx"].score_motion_batch(s["cur"], s["ref"], c["w"], c["h"], s["x0"], s["y0"], c["block"],
                                                 c["block"], c["stride"], c["bilinear"], False, int(c["satd"]), s["cand"])
    if not ok:
        raise RuntimeError(err)
    return costs


def _p_core(s):
    ctx, p = s["ctx"], s["p"]
    ctx.upload_frame(1, *s["cur"])
    a = ctx.analyze_p_core(p, 1, 0, MV_QPEL, False)
    b = ctx.analyze_p_core(p, 1, 0, MV_MIXED, True, seed=a.mvs, seed_distant=a)
    return [_analysis(a), _analysis(b)]


def _p_picture(s):
    ctx, p = s["ctx"], s["p"]
    score = ctx.scene_change_score(p, 1, 0)
    info = ctx.analyze_p_picture(p, s["cfg"], 1, 0, 0, 10, 10)
    out = _analysis(ctx.read_result(p, 0))
    out["scene"] = score
    out["decision"] = np.array([info.mode, info.weighted, info.motion_bits, *info.ic.as_tuple(), *info.cand_bits], np.int64)
    out["scores"] = np.array(list(info.cand_score))
    return out


def _b_picture(s):
    c = s["case"]
    return _analysis(s["ctx"].analyze_b_picture(s["p"], 1, 0, 3, *s["anchor"], c["num"], c["den"],
                                                MV_HPEL_BILINEAR if c["bilinear"] else MV_QPEL))


def _gop(s):
    ctx, p = s["ctx"], s["p"]
    pics, bpics = s["pics"], s["bpics"]
    n = len(pics)
    bslot = lambda k, j, f: 200 + 4 * k + 2 * j + f  # noqa: E731
    ctx.core_passes(p, [(t, r, MV_QPEL, 0, -1, i) for i, (t, r) in enumerate(pics)] +
                    [(t, ref, m, 0, -1, bslot(k, j, f)) for k, (t, past, fut, _n, _d, _a) in enumerate(bpics)
                     for j, m in enumerate((MV_QPEL, MV_HPEL_BILINEAR)) for f, ref in enumerate((past, fut))])
    ctx.core_passes(p, [(t, r, m, 0, i, 20 + 4 * i + j) for i, (t, r) in enumerate(pics) for j, m in enumerate(MODES)])
    ctx.core_passes(p, [(t, r, MV_MIXED, 1, 20 + 4 * i + 2, 100 + i) for i, (t, r) in enumerate(pics)])
    for i, (t, r) in enumerate(pics):
        ctx.motion_compensate(p, r, 100 + i, MV_MIXED, 100 + i)
        ctx.forward_quant_device(p, t, 100 + i, 15, 0, s["levels"][i].data_ptr())
    if bpics:
        ctx.b_decide(p, [(t, past, fut, bslot(k, j, 0), bslot(k, j, 1), 100 + a, num, den, m, 2 * k + j)
                         for k, (t, past, fut, num, den, a) in enumerate(bpics)
                         for j, m in enumerate((MV_QPEL, MV_HPEL_BILINEAR))])
    ic = ctx.estimate_intensity_batch(p, [(t, r, 100 + i) for i, (t, r) in enumerate(pics)])
    out = dict(p=_analyses(s, "p_out", [ctx.read_result(p, 100 + i) for i in range(n)]), ic=np.array(ic, np.int32),
               levels=s["levels"])
    if bpics:
        out["b"] = _analyses(s, "b_out", [ctx.read_bresult(p, k) for k in range(2 * len(bpics))])
    return out


def _clips(s):
    ctx = s["ctx"]
    ctx.core_passes_multi(s["params"], s["passes"])
    return _analyses(s, "out", [ctx.read_result(s["params"][i], s["passes"][i][5]) for i in range(len(s["passes"]))])


def _longrange(s):
    ctx, p, n = s["ctx"], s["p"], s["case"]["pictures"]
    ctx.core_passes(p, [(2 * k + 1, 2 * k, MV_QPEL, 0, -1, k) for k in range(n)])
    return _analyses(s, "out", [ctx.read_result(p, k) for k in range(n)])


def _transform(s):
    ctx, p = s["ctx"], s["p"]
    if s["case"]["dquant"]:
        d, mq, lv = ctx.choose_dquant(p, s["cfg"], 1, 2, s["base"])
        out = dict(mquant=mq)
    else:
        d, lv = ctx.choose_transform(p, s["cfg"], 1, 2)
        out = {}
    out.update({n: d[n] for n in TDECISION_DTYPE.names if n != "reserved"})
    out["levels"] = lv
    return out


def _recon(s):
    ctx, p, c = s["ctx"], s["p"], s["case"]
    ctx.forward_quant_device(p, 1, 2, 15, s["coeffs"].data_ptr() if c["coeffs"] else 0, s["levels"].data_ptr())
    ctx.reconstruct(p, 2, s["levels"].data_ptr(), 15, s["types"], 3)
    ctx.loop_filter(p, 3, *s["meta"])
    out = dict(frame=list(ctx.download_frame(3, c["w"], c["h"])), levels=s["levels"])
    if c["coeffs"]:
        out["coeffs"] = s["coeffs"]
    return out


def _intra(s):
    ctx, p = s["ctx"], s["p"]
    mbw, mbh = mbs_of(p)
    d = [t.data_ptr() for t in s["planes"]]
    mode, flags = ctx.choose_i_overlap(p, 0, cfg=s["cfg"])
    ctx.reconstruct_intra(p, 0, *d, overlap=mode, flags=flags if mode == 2 else None, cfg=s["cfg"])
    if mode:
        ctx.overlap_smooth(p, *d, flags=flags if mode == 2 else None, all_edges=mode == 1)
    ctx.store_signed(p, *d, 128, 1)
    ctx.loop_filter(p, 1)
    return dict(mode=mode, flags=flags, frame=list(ctx.download_frame(1, 16 * mbw, 16 * mbh)), planes=s["planes"])


def _learned(s):
    ctx, p, net, n = s["ctx"], s["p"], s["net"], s["case"]["pairs"]
    for k in range(n):
        net.prepare(2 * k, 2 * k + 1, k)
    net.propose(0, n)
    net.analyze(p, [(2 * k, 2 * k + 1, k, MV_QPEL, 100 + k) for k in range(n)], fallback=True)
    return _analyses(s, "out", [ctx.read_result(p, 100 + k) for k in range(n)])


def _train(s):
    loss, grads = s["net"].gradients(list(range(s["case"]["pairs"])))
    return [np.float32(loss), grads]


_RUN = dict(score=_score, p_core=_p_core, p_picture=_p_picture, b_picture=_b_picture, gop=_gop, clips=_clips,
            longrange=_longrange, transform=_transform, recon=_recon, intra=_intra, learned=_learned, train=_train)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---- what a pass cannot do without ----------------------------------------------------------

# Integer operations per macroblock of the passes, counted by the instrumented oracle on the 1080p
# GOP (search range 64), and of the four transform sizes' matrices; a window's share scales with the
# searched candidates, the rest does not.
_OPS = dict(unseeded=286137, b_pass=205000, mode_passes=56261 + 25322 + 471920, final=472179, xform=51912)
_ROW = 96  # bytes of one macroblock's result


def work(case):
    kind = case["kind"]
    if kind == "score":
        b, n = case["block"], case["n"]
        return dict(bytes=float(b * b + (b + 131) ** 2 + 16 * n), flops=float(n * b * b * 3))
    if kind == "clips":
        mbs = sum(((w + 15) // 16) * ((h + 15) // 16) for w, h, _ in _clip_sizes(case))
        return dict(bytes=float(mbs * (2 * 256 + 5 * _ROW)),
                    flops=float(mbs * (_OPS["unseeded"] + _OPS["mode_passes"] + _OPS["final"])))
    mbs = ((case["w"] + 15) // 16) * ((case["h"] + 15) // 16)
    px = mbs * 384  # 4:2:0 bytes of a picture
    if kind == "p_core":
        return dict(bytes=float(2 * px + 2 * mbs * _ROW), flops=float(mbs * (_OPS["unseeded"] + _OPS["final"])))
    if kind == "p_picture":
        return dict(bytes=float(2 * px + mbs * _ROW),
                    flops=float(mbs * (_OPS["unseeded"] + _OPS["mode_passes"] + _OPS["final"])))
    if kind == "b_picture":
        return dict(bytes=float(3 * px + mbs * _ROW), flops=float(mbs * 2 * _OPS["unseeded"]))
    if kind == "gop":
        n = case["frames"]
        np_ = -(-(n - 1) // 3)
        nb = n - 1 - np_
        return dict(bytes=float(n * px + np_ * mbs * (_ROW + 4 * 768) + nb * mbs * 2 * _ROW),
                    flops=float(mbs * (np_ * (_OPS["unseeded"] + _OPS["mode_passes"] + _OPS["final"] + _OPS["xform"]) +
                                       nb * 4 * _OPS["b_pass"])))
    if kind == "longrange":
        return dict(bytes=float(case["pictures"] * (2 * px + mbs * _ROW)),
                    flops=float(case["pictures"] * mbs * _OPS["unseeded"]))
    if kind == "transform":
        return dict(bytes=float(2 * px + mbs * (768 + TDECISION_DTYPE.itemsize)), flops=float(mbs * 4 * _OPS["xform"]))
    if kind == "recon":
        extra = 4 * mbs * 384 * 8 if case["coeffs"] else 0
        return dict(bytes=float(3 * px + 4 * mbs * 768 + extra), flops=float(mbs * (_OPS["xform"] + 384 * 16)))
    if kind == "intra":
        return dict(bytes=float(2 * px + px * 4), flops=float(mbs * 6 * 8 * 8 * 8 * 4))
    q = mbs * 16  # samples of the quarter-resolution picture
    net = 2.0 * q * 9 * 32 * (16 + 3 * 32)
    if kind == "learned":
        return dict(bytes=float(case["pairs"] * (2 * px + mbs * _ROW)), flops=float(case["pairs"] * (net + mbs * 60000)))
    return dict(bytes=float(case["pairs"] * (q * 32 + mbs * 8) + 2 * 32648 * 4), flops=float(case["pairs"] * 3 * net))


# ---- values in 64 bits ----------------------------------------------------------------------

_K4 = np.array([[0.0147058823529412] * 4,
                [0.0188356164383562, 0.0085616438356164, -0.0085616438356164, -0.0188356164383562],
                [0.0147058823529412, -0.0147058823529412, -0.0147058823529412, 0.0147058823529412],
                [0.0085616438356164, -0.0188356164383562, 0.0188356164383562, -0.0085616438356164]])
_A, _B, _C, _D, _E, _F, _G = (0.010416666667, 0.013840830450, 0.012975778547, 0.007785467128, 0.003460207612,
                              0.013698630137, 0.005136986301)
_K8 = np.array([[_A] * 8, [_B, _C, _D, _E, -_E, -_D, -_C, -_B], [_F, _G, -_G, -_F, -_F, -_G, _G, _F],
                [_C, -_E, -_B, -_D, _D, _B, _E, -_C], [_A, -_A, -_A, _A, _A, -_A, -_A, _A],
                [_D, -_B, _E, _C, -_C, -_E, _B, -_D], [_G, -_F, _F, -_G, -_G, _F, -_F, _G],
                [_E, -_D, _C, -_B, _B, -_C, _D, -_E]])


_OFF_SCALE, _OFF_CLIP = 4.0, 4.0  # pixels per unit of a regressed offset; its largest value


def _exact_coeffs(case, seed):
    """The four transform sizes' coefficients of the residual, [type][mb][parent][64]."""
    s = prepare(case, seed)
    w, h = case["w"], case["h"]
    src, pred = s["ctx"].download_frame(1, w, h), s["ctx"].download_frame(2, w, h)
    mbw, mbh = mbs_of(s["p"])
    out = np.zeros((4, mbw * mbh, 6, 64))
    for pl in range(3):
        r = src[pl].astype(np.float64) - pred[pl].astype(np.float64)
        ph, pw = r.shape
        n = 2 if pl == 0 else 1
        full = np.zeros((8 * n * mbh, 8 * n * mbw))
        full[:ph, :pw] = r
        blocks = full.reshape(mbh, n, 8, mbw, n, 8).transpose(0, 3, 1, 4, 2, 5).reshape(mbw * mbh, n * n, 8, 8)
        dst = slice(0, 4) if pl == 0 else slice(3 + pl, 4 + pl)
        # a partition that lies wholly outside the raster codes nothing; its residual is zero already
        out[0, :, dst] = (1024.0 * (_K8 @ blocks @ _K8.T)).transpose(0, 1, 3, 2).reshape(mbw * mbh, n * n, 64)
        for t, (bh, bw) in ((1, (4, 8)), (2, (8, 4)), (3, (4, 4))):
            kv, kh = (_K8 if bh == 8 else _K4), (_K8 if bw == 8 else _K4)
            o = np.zeros_like(blocks)
            for y in range(0, 8, bh):
                for x in range(0, 8, bw):
                    o[..., y:y + bh, x:x + bw] = 1024.0 * (kv @ blocks[..., y:y + bh, x:x + bw] @ kh.T)
            out[t, :, dst] = o.reshape(mbw * mbh, n * n, 64)
    s["ctx"].close()
    return out


def _exact_train(case, seed):
    """The network's mean loss and its gradients in float64 (3x3 convolutions with ReLU over the 16
    input features, the mean of a macroblock's samples, two logistic and two offset terms)."""
    s = prepare(case, seed)
    ctx, net, p, n = s["ctx"], s["net"], s["p"], case["pairs"]
    mbw, mbh = mbs_of(p)
    feats, hints, labels = [], [], []
    for k in range(n):
        f, hint, _c, _fb = net.read_sample(k)
        feats.append(torch.from_numpy(f.view(np.int16).copy()).view(torch.bfloat16).double())
        hints.append(torch.from_numpy(hint.astype(np.float64)))
        labels.append(torch.from_numpy(((ctx.read_result(p, k).mvs.astype(np.int64) + 2) >> 2).astype(np.float64)))
    theta = torch.from_numpy(net.params().astype(np.float64)).cuda().requires_grad_(True)
    x = torch.stack(feats).cuda()
    pos = 0

    def take(*shape):
        nonlocal pos
        m = int(np.prod(shape))
        pos += m
        return theta[pos - m:pos].reshape(shape)

    for cin in (16, 32, 32, 32):
        wt, b = take(32, 9, cin), take(32)
        pad = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
        hh, ww = x.shape[1], x.shape[2]
        z = b.expand(n, hh, ww, 32)
        for tap in range(9):
            z = z + pad[:, tap // 3:tap // 3 + hh, tap % 3:tap % 3 + ww] @ wt[:, tap].T
        x = torch.relu(z)
    wh, bh = take(8, 32), take(8)
    pooled = x.reshape(n, mbh, 4, mbw, 4, 32).mean(dim=(2, 4)).reshape(n, mbh * mbw, 32)
    out = pooled @ wh.T + bh
    loss = 0.0
    for f in range(n):
        lab, o = labels[f].cuda(), out[f]
        hyp = [torch.zeros(2, dtype=torch.float64, device="cuda"), hints[f].cuda()]
        near = ((lab - hyp[0]).abs().sum(1) > (lab - hyp[1]).abs().sum(1)).double()
        for k in range(2):
            tgt = near if k else 1.0 - near
            loss = loss + (torch.nn.functional.softplus(o[:, k], threshold=1e9) - tgt * o[:, k]).sum()
            d = lab - hyp[k]
            mask = (d.abs().amax(1) <= _OFF_SCALE * _OFF_CLIP).double()
            e = o[:, 2 + 2 * k:4 + 2 * k] - (d / _OFF_SCALE).clamp(-_OFF_CLIP, _OFF_CLIP)
            sl = torch.where(e.abs() < 1.0, 0.5 * e * e, e.abs() - 0.5)
            loss = loss + (sl.sum(1) * mask).sum()
    loss = loss / (n * mbw * mbh)
    loss.backward()
    res = [float(loss.detach()), theta.grad.cpu().numpy()]
    net.close()
    ctx.close()
    return res


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "recon" and case["coeffs"]:
        return dict(frame=[None, None, None], levels=None, coeffs=_exact_coeffs(case, seed))
    return None
