"""The work that users of this package have it do, as cases that can be timed and
checked: playback (decoding), the encoder's stages (registration, fitting
clouds, colour interpolation, colour coding, quality), zstd payloads, and the
registration network's training.  Each case goes through the package's public
calls; inputs come from the package's seeded synthetic sequences at the sizes
of its configurations, tests and benchmark.

  listed()               the named cases
  draw(rng)              one more case of the same ranges
  prepare(case, seed)    inputs, and the plan or handle a program keeps
  run(state)             one pass and its outputs
  work(case)             bytes and operations one pass cannot do without
  exact(case, seed)      what run returns, in 64 bits, by plain numpy / torch
"""
from __future__ import annotations

import ctypes
import math
import os
import struct
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "patchvvc-plus_gb300"))

import pvvc  # noqa: E402
from pvvc import _lib  # noqa: E402
from pvvc.fitting import Fitter  # noqa: E402
from pvvc.icp import IcpBatch, KnnColorBatch, make_pairs_packed  # noqa: E402
from pvvc.quality import Quality  # noqa: E402
from pvvc.regnet import DIMS, RegNet  # noqa: E402

DEV = "cuda"

# Sequences: "tiny" (2.7k points a frame on a 128^3 grid), "gof8" (100k points a
# frame, 9 bits, 60 patches of 800-2500) and "seq300" (10 bits, lognormal
# patches of 200-8000, median 1500; `points` a frame) are the package's own
# workloads.


def listed():
    return [
        # a viewer that opens a very small clip: call latency counts
        dict(name="host_tiny", kind="host", seq="tiny", frames=4, gof=4, points=3000, qp=8, zstd=0, pinned=False),
        # a client that decodes a GoF of 8 frames from .frame files written with
        # the reference's zstd level, into page-locked arrays
        dict(name="host_gof8_zstd", kind="host", seq="gof8", frames=8, gof=8, points=115000, qp=8, zstd=22, pinned=True),
        # the same GoF with its payloads on the device, one graph launch
        dict(name="plan_gof8", kind="plan", seq="gof8", frames=8, gof=8, points=115000, streams=1, qp=8),
        # what the playback server decodes at once: a few streams' next frames
        dict(name="plan_streams", kind="plan", seq="seq300", frames=2, gof=30, points=500000, streams=4, qp=8),
        # a whole GoP of 30 frames of ~800k points (10-bit sequence)
        dict(name="plan_gop30", kind="plan", seq="seq300", frames=30, gof=30, points=920000, streams=1, qp=8),
        # a GoP's level-22 payloads inflated on the device
        dict(name="inflate_gop", kind="inflate", frames=30, points=920000, level=22),
        # one frame's patches registered onto the fitting clouds
        dict(name="icp_frame", kind="icp", pairs=472, deg=15.0, trans=20.0, max_iter=50),
        # a GoP's colours interpolated onto the fitting clouds (10 neighbours),
        # later frames as residuals
        dict(name="knn_gop", kind="knn", points=230000, frames=30, k=10),
        # a decoded frame measured against its source
        dict(name="quality_frame", kind="quality", points=920000, jitter=0.3),
        # fitting clouds of 40 patches over a GoP of 30 frames
        dict(name="fit_patches", kind="fit", patches=40, frames=30),
        # the colour payloads of a GoP from the leaf colours
        dict(name="encode_gop", kind="encode", points=230000, frames=30, qp=8),
        # one batch's loss and gradient in the registration network's training
        dict(name="train_grad", kind="grad", batch=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "plan", "plan", "plan", "inflate", "icp", "icp", "knn", "quality", "fit", "encode", "grad"])
    if kind == "host":
        seq = rng.choice(["tiny", "gof8", "seq300"])
        pts = {"tiny": _log(rng, 1000, 9000), "gof8": _log(rng, 20000, 115000), "seq300": _log(rng, 30000, 200000)}[seq]
        frames = rng.randint(1, 8)
        return dict(kind=kind, seq=seq, frames=frames, gof=rng.choice([4, 8, 30]), points=pts, qp=rng.choice([4, 8, 16, 32]),
                    zstd=rng.choice([0, 0, 22]), pinned=rng.random() < 0.5)
    if kind == "plan":
        # one GoP of one stream, or the next frames of several streams
        if rng.random() < 0.5:
            frames = rng.randint(3, 30)
            return dict(kind=kind, seq=rng.choice(["gof8", "seq300"]), frames=frames, gof=30,
                        points=_log(rng, 60000, 800000), streams=1, qp=rng.choice([4, 8, 16, 32]))
        return dict(kind=kind, seq="seq300", frames=rng.randint(1, 3), gof=30, points=_log(rng, 100000, 500000),
                    streams=rng.randint(2, 8), qp=rng.choice([4, 8, 16, 32]))
    if kind == "inflate":
        return dict(kind=kind, frames=rng.randint(2, 30), points=_log(rng, 50000, 900000), level=rng.choice([3, 9, 22]))
    if kind == "icp":
        # a patch's frames up to a frame's patches; small motion between
        # consecutive frames, or the registration workload's large motion
        deg, trans = rng.choice([(3.0, 2.0), (15.0, 20.0)])
        return dict(kind=kind, pairs=_log(rng, 5, 450), deg=deg, trans=trans, max_iter=rng.choice([10, 30, 50]))
    if kind == "knn":
        return dict(kind=kind, points=_log(rng, 20000, 220000), frames=rng.randint(2, 30), k=rng.choice([1, 4, 10, 16]))
    if kind == "quality":
        return dict(kind=kind, points=_log(rng, 30000, 900000), jitter=round(rng.uniform(0.1, 0.8), 3))
    if kind == "fit":
        return dict(kind=kind, patches=rng.randint(2, 38), frames=rng.choice([8, 15, 30]))
    if kind == "encode":
        return dict(kind=kind, points=_log(rng, 30000, 220000), frames=rng.randint(1, 30), qp=rng.choice([4, 8, 16, 32]))
    return dict(kind="grad", batch=64 * rng.randint(1, 16))


# ---------------------------------------------------------------- inputs

# Sequences of another seed have other patches and point counts.  A program
# keeps its output buffers for sequences of any count up to a limit; so do the
# cases (what lies beyond a sequence's own outputs stays zero).


def _most_points(c):
    return c["points"] * c.get("frames", 1) * c.get("streams", 1)


def _most_slices(c):
    per = c["points"] // 150 + 4 if c.get("seq") == "tiny" else c["points"] // 1200 + 8
    return per * c.get("frames", 1) * c.get("streams", 1)


def _padded(v, n):
    """v followed by zero rows up to n rows (numpy or torch)."""
    if isinstance(v, torch.Tensor):
        return torch.cat([v, v.new_zeros((n - v.shape[0],) + tuple(v.shape[1:]))])
    return np.concatenate([v, np.zeros((n - v.shape[0],) + v.shape[1:], v.dtype)])


def _synth(c, seed, **over):
    k = dict(seed=seed, target_points=c["points"], nframes=c.get("frames", 1), gof=c.get("gof", c.get("frames", 1)))
    if "qp" in c:
        k.update(qp_i=c["qp"], qp_p=c["qp"])
    k.update(over)
    return pvvc.Synth(pvvc.config(c.get("seq", "seq300"), **k))


def _pool(fn, n):
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 4)) as ex:
        return list(ex.map(fn, range(n)))


def _decode_frames(c, seed):
    """One list of .frame bytes per stream."""
    return [_synth(c, 1000 * seed + i, zstd_level=c.get("zstd", 0)).frames() for i in range(c.get("streams", 1))]


def _up(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _moved_patches(c, seed, npatch=None):
    """Per patch: its geometry, and per frame the patch moved by up to a voxel,
    a tenth of its points dropped, with the frame's RGB."""
    syn = _synth(c, seed)
    n = syn.patch_count(0)
    n = n if npatch is None else min(n, npatch)

    def one(p):
        xyz, yuv, _ = syn.patch(0, p)
        rng = np.random.default_rng([seed, p])
        src, col = [], []
        for f in range(yuv.shape[0]):
            keep = rng.random(xyz.shape[0]) > 0.1
            keep[0] = True
            src.append(np.round(xyz[keep] + rng.integers(-1, 2, (int(keep.sum()), 3))).astype(np.float32))
            col.append(np.clip(yuv[0][keep] if f == 0 else yuv[0][keep] + yuv[f][keep], 0, 255).astype(np.uint8))
        return xyz.astype(np.float32), src, col

    return _pool(one, n)


def _knn_inputs(c, seed):
    queries, query_of, sources, rgbs, base = [], [], [], [], []
    for p, (xyz, src, col) in enumerate(_moved_patches(c, seed)):
        first = len(sources)
        for f in range(len(src)):
            query_of.append(p)
            base.append(-1 if f == 0 else first)
        sources += src
        rgbs += col
        queries.append(xyz)
    return queries, query_of, sources, rgbs, base


def _fit_inputs(c, seed):
    """Registered patches: each frame's patch moved, jittered, voxelised and
    brought back by the true motion."""
    syn = _synth(dict(points=8000 + 2400 * c["patches"], frames=c["frames"]), seed)
    n = c["patches"]

    def one(p):
        xyz, _, mv = syn.patch(0, p)
        rng = np.random.default_rng([seed, p])
        pats = [xyz.astype(np.float32)]
        for f in range(1, c["frames"]):
            m = mv[f].astype(np.float64)
            v = np.round(xyz.astype(np.float64) @ m[:3, :3].T + m[:3, 3] + rng.normal(0, 0.3, xyz.shape))
            v = np.unique(v, axis=0)
            inv = np.linalg.inv(m)
            pats.append((v @ inv[:3, :3].T + inv[:3, 3]).astype(np.float32))
        return pats

    return _pool(one, n)


def _most_fit(c):
    return 4000 * c["patches"] + 40000


def _quality_inputs(c, seed):
    """A source frame and its decoded frame: the points jittered and rounded to
    the grid, a few lost, the colours off by a few steps."""
    syn = _synth(dict(points=c["points"]), seed)
    parts = _pool(lambda p: syn.patch(0, p)[:2], syn.patch_count(0))
    rng = np.random.default_rng(seed)
    a = np.concatenate([x for x, _ in parts]).astype(np.float32)
    ca = np.clip(np.concatenate([y[0] for _, y in parts]), 0, 255).astype(np.uint8)
    keep = rng.random(a.shape[0]) > 0.02
    b = np.round(a[keep] + rng.normal(0, c["jitter"], (int(keep.sum()), 3))).astype(np.float32)
    cb = np.clip(ca[keep].astype(np.int32) + rng.integers(-4, 5, (b.shape[0], 3)), 0, 255).astype(np.uint8)
    return a, ca, b, cb


def _grad_inputs(c, seed):
    """Normalised samples of pairs of surface patches, and their targets."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    B, P = c["batch"], 256
    uv = torch.rand(B, P, 2, generator=g, device=DEV) * 2 - 1
    curv = torch.rand(B, 1, 2, generator=g, device=DEV) - 0.5
    src = torch.cat([uv, (curv * uv * uv).sum(2, keepdim=True)], 2)
    w = (torch.rand(B, 3, generator=g, device=DEV) * 2 - 1) * 0.15
    tgt = src + torch.cross(w[:, None].expand(-1, P, -1), src, dim=2) + 0.02 * torch.randn(B, P, 3, generator=g, device=DEV)
    x = torch.stack([src, tgt], 1)
    x = x - x.mean(2, keepdim=True)
    s = x[:, :1].square().sum(3).mean(2).sqrt()[..., None, None]
    y = torch.cat([w, 0.1 * torch.randn(B, 3, generator=g, device=DEV)], 1)
    return (x / s).contiguous(), y.contiguous()


# ---------------------------------------------------------------- prepare and run


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_host(c, seed):
    frames = _decode_frames(c, seed)[0]
    heads = [_read_frame(b) for b in frames]
    most = max(int(h["size"].max()) for h in heads)
    dec = pvvc.Decoder(nslots=max(int(h["index"].max()) for h in heads) + 1, max_leaves=most, max_nodes=2 * most + 64)
    n = _most_points(c)
    out = [torch.zeros((n, 3), dtype=t, pin_memory=c["pinned"]) for t in (torch.float32, torch.uint8)]
    return dict(kind="host", dec=dec, frames=frames, keep=out, out=[t.numpy() for t in out],
                status=np.zeros(_most_slices(c), np.int32))


def _run_host(s):
    _, _, st = s["dec"].decode_frames(s["frames"], out=s["out"])
    s["status"][:st.size] = st
    return s["out"] + [s["status"]]


def _prepare_plan(c, seed):
    packed = [pvvc.pack_frames([pvvc.parse_frame(b) for b in f]) for f in _decode_frames(c, seed)]
    stride = max(int(b.slot.max()) + 1 for b in packed)
    batch = pvvc.concat_batches(packed, slot_stride=stride)
    most = int(batch.size.max())
    dec = pvvc.Decoder(nslots=stride * len(packed), max_leaves=most, max_nodes=2 * most + 64)
    plan = pvvc.Plan(batch)
    n = _most_points(c)
    pay = _up(batch.payload)
    xyz = torch.zeros((n, 3), dtype=torch.float32, device=DEV)
    rgb = torch.zeros((n, 3), dtype=torch.uint8, device=DEV)
    st = torch.zeros(_most_slices(c), dtype=torch.int32, device=DEV)
    ws = torch.empty(max(plan.workspace_bytes, 256), dtype=torch.uint8, device=DEV)
    g = plan.graph(dec, pay.data_ptr(), xyz.data_ptr(), rgb.data_ptr(), 0, st.data_ptr(), ws.data_ptr(), ws.numel())
    return dict(kind="plan", graph=g, keep=(dec, plan, pay, ws), out=[xyz, rgb, st])


def _run_plan(s):
    s["graph"].launch(torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _prepare_inflate(c, seed):
    syn = _synth(dict(points=c["points"], frames=c["frames"]), seed, zstd_level=c["level"])
    jobs = []
    for b in syn.frames():
        f = pvvc.parse_frame(b)
        for i in np.flatnonzero(f.type & 0x18):
            if f.type[i] & 0x08:
                jobs.append(f.geometry[i])
            if f.type[i] & 0x10:
                jobs.append(f.color[i])
    n = len(jobs)
    ln = np.array([len(p) for p in jobs], np.uint32)
    cap = np.array([pvvc.zstd.content_size(p) for p in jobs], np.uint32)
    starts = lambda v: np.concatenate([[0], np.cumsum(v.astype(np.uint64))[:-1]]).astype(np.uint64)  # noqa: E731
    src = _up(np.frombuffer(b"".join(jobs) + b"\0", np.uint8).copy())
    dst = torch.zeros(2 * _most_points(c) + 4096, dtype=torch.uint8, device=DEV)
    so, do = _up(starts(ln).view(np.int64)), _up(starts(cap).view(np.int64))
    ln, cap = _up(ln.view(np.int32)), _up(cap.view(np.int32))
    olen, st = (torch.zeros(2 * _most_slices(c), dtype=torch.int32, device=DEV) for _ in range(2))
    p = [ctypes.c_void_p(t.data_ptr()) for t in (src, so, ln, dst, do, cap, olen, st)]
    return dict(kind="inflate", n=n, ptrs=p, keep=(src, so, ln, do, cap), out=[dst, olen, st])


def _run_inflate(s):
    _lib.check(pvvc.lib().pvvc_zstd_inflate_batch(s["n"], *s["ptrs"], torch.cuda.current_stream().cuda_stream), "inflate")
    return s["out"]


def _prepare_icp(c, seed):
    syn = pvvc.Synth(pvvc.config("seq300", nframes=1, gof=1, seed=seed))
    src, so, tgt, to, _ = make_pairs_packed(c["pairs"], seed=seed, max_deg=c["deg"], max_trans=c["trans"], synth=syn)
    return dict(kind="icp", batch=IcpBatch(None, packed=(src, so, tgt, to)), max_iter=c["max_iter"])


def _run_icp(s):
    b = s["batch"]
    b.run(max_iter=s["max_iter"])
    return [b.T, b.mse, b.iters, b.conv]


def _prepare_knn(c, seed):
    queries, query_of, sources, rgbs, base = _knn_inputs(c, seed)
    b = KnnColorBatch(queries, query_of, sources, rgbs, k=c["k"], base=base)
    b.yuv = torch.zeros((_most_points(c), 3), dtype=torch.float32, device=DEV)
    b.status = torch.zeros(_most_slices(c), dtype=torch.int32, device=DEV)
    return dict(kind="knn", batch=b)


def _run_knn(s):
    s["batch"].run()
    return [s["batch"].yuv, s["batch"].status]


def _prepare_quality(c, seed):
    return dict(kind="quality", q=Quality(), clouds=[_up(v) for v in _quality_inputs(c, seed)])


def _run_quality(s):
    return s["q"].mse(*s["clouds"])


def _prepare_fit(c, seed):
    gops = _fit_inputs(c, seed)
    return dict(kind="fit", fitter=Fitter(), gops=gops, seeds=np.arange(1, len(gops) + 1, dtype=np.uint32),
                out=np.zeros((_most_fit(c), 3), np.float32))


def _run_fit(s):
    clouds, _ = s["fitter"].fit(s["gops"], seeds=s["seeds"])
    size = np.array([v.shape[0] for v in clouds])
    np.concatenate(clouds, out=s["out"][:size.sum()])
    return [s["out"], size]


def _prepare_encode(c, seed):
    syn = _synth(dict(points=c["points"], frames=c["frames"]), seed)
    n = syn.patch_count(0)

    def one(p):
        xyz, yuv, _ = syn.patch(0, p)
        return pvvc.patch_leaf_yuv(xyz, yuv)

    parts = _pool(one, n)
    size = np.array([k for _, k, _ in parts], np.uint32)
    frames = [pvvc.Frame(f, np.arange(n, dtype=np.int32), np.full(n, 3 if f else 1, np.uint8), size,
                         np.full(n, c["qp"], np.uint8), np.tile(np.eye(4, dtype=np.float32).reshape(16), (n, 1)),
                         [b"" if f else g for g, _, _ in parts], [b""] * n) for f in range(c["frames"])]
    batch = pvvc.pack_frames(frames)
    leaf = np.concatenate([parts[p][2][f] for f in range(c["frames"]) for p in range(n)])
    cap = ((16 * batch.size.astype(np.uint64) + 64 + 3) // 4 * 4).astype(np.uint32)
    off = np.concatenate([[0], np.cumsum(cap.astype(np.uint64))[:-1]]).astype(np.uint64)
    out = torch.zeros(17 * _most_points(c) + 68 * _most_slices(c), dtype=torch.uint8, device=DEV)
    olen, st = (torch.zeros(_most_slices(c), dtype=torch.int32, device=DEV) for _ in range(2))
    most = int(size.max())
    return dict(kind="encode", enc=pvvc.Encoder(), dec=pvvc.Decoder(nslots=n, max_leaves=most, max_nodes=2 * most + 64),
                batch=batch, pay=_up(batch.payload), leaf=_up(leaf), off=off, cap=cap, out=[out, olen, st])


def _run_encode(s):
    out, olen, st = s["out"]
    s["enc"].encode(s["batch"], s["dec"], s["pay"].data_ptr(), s["leaf"].data_ptr(), out.data_ptr(), s["off"], s["cap"],
                    olen.data_ptr(), st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _prepare_grad(c, seed):
    x, y = _grad_inputs(c, seed)
    return dict(kind="grad", net=RegNet(seed=seed), x=x, y=y)


def _run_grad(s):
    return list(s["net"].grad(s["x"], s["y"], 10.0, stream=torch.cuda.current_stream().cuda_stream))


_PREPARE = dict(host=_prepare_host, plan=_prepare_plan, inflate=_prepare_inflate, icp=_prepare_icp, knn=_prepare_knn,
                quality=_prepare_quality, fit=_prepare_fit, encode=_prepare_encode, grad=_prepare_grad)
_RUN = dict(host=_run_host, plan=_run_plan, inflate=_run_inflate, icp=_run_icp, knn=_run_knn, quality=_run_quality,
            fit=_run_fit, encode=_run_encode, grad=_run_grad)


# ---------------------------------------------------------------- work


def work(case):
    """From the case's sizes (points a frame are near 0.87 of the target)."""
    k = case["kind"]
    if k in ("host", "plan"):
        # payloads in (about 0.6 byte a point), xyz + rgb out (15), the
        # reference colours read once a predictive point (12)
        pts = 0.87 * case["points"] * case["frames"] * case.get("streams", 1)
        return dict(bytes=27.6 * pts, flops=60.0 * pts)
    if k == "inflate":
        pts = 0.87 * case["points"] * case["frames"]
        return dict(bytes=0.7 * pts, flops=0.0)
    if k == "icp":
        # each cloud once; per iteration and source point the transform (18),
        # the distance to its neighbour (8) and the correspondence sums (26)
        pts = 1680.0 * case["pairs"]
        return dict(bytes=12 * 2.05 * pts, flops=52.0 * pts * case["max_iter"])
    if k == "knn":
        q = 0.87 * case["points"] * case["frames"]
        return dict(bytes=0.9 * 15 * q + 12 * q, flops=q * case["k"] * 20)
    if k == "quality":
        return dict(bytes=0.87 * case["points"] * 2 * 15, flops=0.87 * case["points"] * 2 * 40)
    if k == "fit":
        pts = 1600.0 * case["patches"] * case["frames"]
        return dict(bytes=12 * pts, flops=8 * pts)
    if k == "encode":
        pts = 0.87 * case["points"] * case["frames"]
        return dict(bytes=12.6 * pts, flops=60.0 * pts)
    # grad: both clouds' points in, one gradient out; layers 2 and 3 per
    # sampled point forward, layer 2 backward (the pooled layer 3 is sparse),
    # the head per pair
    rows = 512.0 * case["batch"]
    return dict(bytes=12 * rows + 4 * 208000, flops=2 * rows * (3 * 64 * 2 + 64 * 128 * 3 + 128 * 256) + 6.0 * case["batch"] * 164608)


# ---------------------------------------------------------------- exact


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None


def _read_frame(b):
    """The .frame layout: header arrays, then geometry and colour payloads."""
    _, n = struct.unpack_from("<iI", b, 0)
    o = [8]

    def take(dt, m):
        a = np.frombuffer(b, dt, m, o[0])
        o[0] += a.nbytes
        return a

    f = dict(n=n, index=take("<i4", n), type=take("u1", n), size=take("<u4", n), qp=take("u1", n),
             mv=take("<f4", 16 * n).reshape(n, 4, 4))
    f["geo"] = []
    for g in take("<u4", n):
        f["geo"].append(b[o[0]:o[0] + int(g)])
        o[0] += int(g)
    return f


def _leaf_centres(geo):
    """Leaf centres of one patch's octree, breadth first, in 64 bits."""
    head = np.frombuffer(geo, ">f4", 6).astype(np.float64)
    ctr, rng, h = head[None, :3], head[3:], geo[24]
    occ, at = np.frombuffer(geo, np.uint8), 25
    bit = np.arange(8)
    sign = np.stack([np.where(bit & 4, -1, 1), np.where(bit & 2, -1, 1), np.where(bit & 1, -1, 1)], 1)
    for _ in range(h - 1):
        rng = rng / 2
        has = (occ[at:at + len(ctr), None] & (0x80 >> bit)[None]) != 0
        at += len(ctr)
        node, child = np.nonzero(has)
        ctr = ctr[node] + sign[child] * (rng / 2)
    return ctr


def _exact_decode(case, seed):
    """The coordinates: each slice's leaf centres by its matrix.  The colours
    are bytes and the statuses whole numbers: they stay equal."""
    if case.get("zstd"):
        return None  # geometry inside zstd frames
    parts = []
    for frames in _decode_frames(case, seed):
        tree = {}
        for b in frames:
            f = _read_frame(b)
            for i in range(f["n"]):
                if not f["type"][i] & 2:
                    tree[int(f["index"][i])] = _leaf_centres(f["geo"][i])
                m = f["mv"][i].astype(np.float64)
                parts.append(tree[int(f["index"][i])] @ m[:3, :3].T + m[:3, 3])
    return [_padded(np.concatenate(parts), _most_points(case)), None, None]


def _exact_knn(case, seed):
    queries, query_of, sources, rgbs, base = _knn_inputs(case, seed)
    K = torch.tensor([[0.299, 0.587, 0.114], [-0.168736, -0.331264, 0.5], [0.5, -0.418688, -0.081312]], dtype=torch.float64,
                     device=DEV)
    qs = [_up(q).double() for q in queries]
    outs = []
    for p, (s, c) in enumerate(zip(sources, rgbs)):
        q, s, c = qs[query_of[p]], _up(s).double(), _up(c).double()
        d = sum((q[:, k:k + 1] - s[None, :, k]) ** 2 for k in range(3))
        dk, ik = torch.topk(d, min(case["k"], s.shape[0]), dim=1, largest=False)
        w = 1 / dk.clamp_min(1e-6)
        rgb = ((w / w.sum(1, keepdim=True))[..., None] * c[ik]).sum(1)
        outs.append(rgb @ K.T + torch.tensor([0.0, 128.0, 128.0], dtype=torch.float64, device=DEV))
    outs = [o if b < 0 else o - outs[b] for o, b in zip(outs, base)]
    return [_padded(torch.cat(outs), _most_points(case)), None]


def _exact_icp(case, seed):
    """Point-to-point ICP by brute force.  Each step's neighbours are a discrete
    choice, so a pair may take another path near a tie."""
    b = _prepare_icp(case, seed)["batch"]
    so, to = b.soff.tolist(), b.toff.tolist()
    T, mse = [], []
    for p in range(b.n):
        s, t = b.src[so[p]:so[p + 1]].double(), b.tgt[to[p]:to[p + 1]].double()
        M, last = np.eye(4), math.inf

        def moved():
            R = torch.from_numpy(M).to(DEV)
            q = s @ R[:3, :3].T + R[:3, 3]
            return (q,) + sum((q[:, k:k + 1] - t[None, :, k]) ** 2 for k in range(3)).min(1)

        for it in range(case["max_iter"]):
            q, d, at = moved()
            m = t[at]
            cq, cm = q.mean(0), m.mean(0)
            h = torch.cat([((q - cq).T @ (m - cm)).reshape(-1), cq, cm, d.mean()[None]]).cpu().numpy()
            U, _, Vt = np.linalg.svd(h[:9].reshape(3, 3))
            R = Vt.T @ np.diag([1, 1, np.sign(np.linalg.det(Vt.T @ U.T))]) @ U.T
            step = np.eye(4)
            step[:3, :3], step[:3, 3] = R, h[12:15] - R @ h[9:12]
            M = step @ M
            if abs(h[15] - last) < 1e-6:
                break
            last = h[15]
        T.append(M.reshape(16))
        mse.append(float(moved()[1].mean()))
    return [np.stack(T), np.array(mse), None, None]


def _exact_quality(case, seed):
    a, ca, b, cb = (_up(v).double() for v in _quality_inputs(case, seed))
    K = torch.tensor([[0.299, 0.587, 0.114], [-0.168736, -0.331264, 0.5], [0.5, -0.418688, -0.081312]], dtype=torch.float64,
                     device=DEV)

    def side(q, qc, t, tc):
        """Nearest neighbours with the query cloud cut into slabs along x, each
        slab against the targets within 12 voxels of it (against all targets
        where a neighbour lies further); the first target among equal ones."""
        ts, tx = torch.sort(t[:, 0], stable=True)
        total = torch.zeros(4, dtype=torch.float64, device=DEV)
        for rows in torch.split(torch.argsort(q[:, 0]), 2048):
            x = q[rows]
            lo, hi = float(x[:, 0].min()), float(x[:, 0].max())
            i0, i1 = (int(torch.searchsorted(ts, torch.tensor(v, dtype=torch.float64, device=DEV))) for v in (lo - 12, hi + 12))
            for near in (tx[i0:i1], tx):
                if not near.numel():
                    continue
                near = near.sort().values
                y = t[near]
                d = sum((x[:, k:k + 1] - y[None, :, k]) ** 2 for k in range(3))
                best = d.min(1).values
                if near.numel() == t.shape[0] or float(best.max()) < 144:
                    break
            at = near[torch.argmax((d == best[:, None]).to(torch.uint8), dim=1)]
            e = (qc[rows] - tc[at]) @ K.T
            total += torch.cat([best.sum()[None], (e * e).sum(0)])
        return (total / q.shape[0]).cpu().numpy()

    return np.stack([side(a, ca, b, cb), side(b, cb, a, ca)], 1).reshape(-1)


def _exact_grad(case, seed):
    x, y = _grad_inputs(case, seed)
    net = RegNet(seed=seed)
    flat = torch.from_numpy(net.get_params()).to(DEV).double().requires_grad_(True)
    net.close()
    par, o = {}, 0
    for k, shape in DIMS.items():
        n = math.prod(shape)
        par[k] = flat[o:o + n].view(shape)
        o += n
    loss = 0
    for xs, ys in zip(torch.split(x, 128), torch.split(y, 128)):
        h = xs.double().reshape(-1, 3)
        for i in (1, 2, 3):
            h = torch.relu(h @ par[f"w{i}"].T + par[f"b{i}"])
        h = h.view(xs.shape[0], 2, 256, 256).amax(2).reshape(xs.shape[0], 512)
        for i in (4, 5):
            h = torch.relu(h @ par[f"w{i}"].T + par[f"b{i}"])
        e = (h @ par["w6"].T + par["b6"] - ys.double()) ** 2
        part = (10.0 * e[:, :3].sum() + e[:, 3:].sum()) / x.shape[0]
        part.backward(retain_graph=True)
        loss += float(part.detach())
    return [flat.grad, torch.tensor([loss], dtype=torch.float64)]


_EXACT = dict(host=_exact_decode, plan=_exact_decode, icp=_exact_icp, knn=_exact_knn, quality=_exact_quality, grad=_exact_grad)
