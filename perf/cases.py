"""Measured cases of the reconstruction engine: what its users run, through the Python entry points.

Every case is one pass of a user's program over inputs it already holds on the GPU:

* ``insert``: one reconstruction -- zeroed volume and weights, then ``FRB200.Execute``.  With
  several ``batches`` it is the streaming loop of the reference's example driver: per batch the
  traverse spaces from the batch's rotations, then one Execute into the same volume.
* ``jobs``: several uneven reconstructions in one ``FRBatch`` launch (captured in a CUDA graph).
* ``serve``: jobs opened on an ``FRServer``, streamed to it in batches, waited for and read.
* ``prep``: projection images to processed half-planes (``Prep``).

Inputs are the seeded phantom projections of ``umpalumpa_b200.synthetic`` at its benchmark's
noise levels.  ``exact`` evaluates the same reconstruction in FP64 with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from umpalumpa_b200 import synthetic
from umpalumpa_b200.fr import (FRB200, BandedPlanes, FRBatch, InputData, OutputData, Prep, Settings, bricks_of,
                               compute_traverse_spaces)
from umpalumpa_b200.server import FRServer

RADIUS = float(np.float32(1.9))  # blob radius of every configuration
ALPHA = 15.0
TABLE = 10000                    # lookup table entries of every configuration
STORAGES = ("fp32", "bf16", "fp16")
MAX_WORK = 20000 * 257.0 ** 2    # projections x volume face of the largest listed insertion


def listed():
    return [
        # the smallest call: a test-sized reconstruction, all launch and planning latency
        {"name": "insert_box32", "kind": "insert", "box": 32, "batches": "64", "interp": "lookup", "type": "precise",
         "storage": "fp32", "kahan": False},
        # the 2,000-projection box-64 reconstruction, streamed in the served trace's batch sizes
        {"name": "stream_box64", "kind": "insert", "box": 64, "batches": "256,731,1013", "interp": "lookup",
         "type": "precise", "storage": "fp32", "kahan": False},
        # one class of a small classification job, 16-bit projections, on-the-fly blob values
        {"name": "insert_box96_fp16_dynamic", "kind": "insert", "box": 96, "batches": "777", "interp": "dynamic",
         "type": "precise", "storage": "fp16", "kahan": False},
        # a streaming client at production size: batches of the served trace's range
        {"name": "stream_box256", "kind": "insert", "box": 256, "batches": "1024,513", "interp": "lookup",
         "type": "precise", "storage": "fp32", "kahan": False},
        # the production reconstruction (largest job of the batched configuration)
        {"name": "insert_box256", "kind": "insert", "box": 256, "batches": "20000", "interp": "lookup",
         "type": "precise", "storage": "fp32", "kahan": False},
        # the same volume without a lookup table (the reference's default interpolation)
        {"name": "insert_box256_dynamic", "kind": "insert", "box": 256, "batches": "6000", "interp": "dynamic",
         "type": "precise", "storage": "fp32", "kahan": False},
        # nearest-pixel insertion (the reference's default type), for quick previews
        {"name": "insert_box256_fast", "kind": "insert", "box": 256, "batches": "8192", "interp": "dynamic",
         "type": "fast", "storage": "fp32", "kahan": False},
        # the reduced-precision configuration: box 384, BF16 projections, compensated sums
        {"name": "insert_box384_bf16_kahan", "kind": "insert", "box": 384, "batches": "4000", "interp": "lookup",
         "type": "precise", "storage": "bf16", "kahan": True},
        # per-class volumes of mixed sizes in one captured launch (the batched configuration's mix)
        {"name": "jobs_mixed", "kind": "jobs",
         "jobs": "96:2210,256:1480,128:3105,192:3001,96:5020,128:911,256:2750,192:1337,96:500,128:7013,192:4100,96:1649",
         "storage": "fp32"},
        # reconstructions streamed to the request loop (the served trace's boxes and batch sizes)
        {"name": "serve_mixed", "kind": "serve", "jobs": "64:2000,96:3100,128:2500,192:2200,256:2048,320:2001",
         "batch": 1024, "storage": "fp32"},
        # input preparation at production size, into the layout the insertion reads
        {"name": "prep_box256", "kind": "prep", "box": 256, "images": 8192, "storage": "fp32", "layout": "banded"},
        # input preparation of a side the engine's own FFT does not cover, 16-bit output
        {"name": "prep_box192_bf16", "kind": "prep", "box": 192, "images": 2999, "storage": "bf16", "layout": "rows"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: even boxes 32..384 (the serving, batched and reduced-precision
    configurations' range) and projection counts spread over their logarithm."""
    kind = rng.choice(["insert"] * 6 + ["jobs", "jobs", "serve", "prep", "prep"])
    if kind == "prep":
        box = rng.choice([64, 96, 128, 192, 256, 256, 320])
        most = int(8192 * 256 * 256 / (box * box))
        return {"kind": kind, "box": box, "images": _log_int(rng, 50, min(most, 20000)),
                "storage": rng.choice(STORAGES), "layout": rng.choice(["rows", "banded"])}
    if kind == "jobs":
        jobs = [f"{rng.choice([64, 96, 128, 192, 256])}:{_log_int(rng, 500, 4000)}" for _ in range(rng.randint(4, 14))]
        return {"kind": kind, "jobs": ",".join(jobs), "storage": rng.choice(["fp32", "fp32", "bf16"])}
    if kind == "serve":
        jobs = [f"{rng.choice(synthetic.SERVED_BOXES)}:{_log_int(rng, 500, 3000)}" for _ in range(rng.randint(2, 7))]
        return {"kind": kind, "jobs": ",".join(jobs), "batch": rng.randint(256, 2048), "storage": "fp32"}
    box = 2 * rng.randint(16, 192)
    most = max(400, int(0.4 * MAX_WORK / (box + 1) ** 2))
    total = _log_int(rng, 40, min(most, 20000))
    batches = []
    if rng.random() < 0.4:  # streamed in batches of uneven sizes
        left = total
        while left > 0 and len(batches) < 6:
            n = min(left, rng.randint(max(1, total // 5), max(2, total // 2)))
            batches.append(n)
            left -= n
    else:
        batches = [total]
    return {"kind": kind, "box": box, "batches": ",".join(map(str, batches)),
            "interp": rng.choice(["lookup", "lookup", "dynamic"]),
            "type": rng.choice(["precise"] * 4 + ["fast"]), "storage": rng.choice(["fp32", "fp32", "bf16", "fp16"]),
            "kahan": rng.random() < 0.25}


# ---- inputs -------------------------------------------------------------------------------

DEV = "cuda"


def _dtype(storage):
    return torch.bfloat16 if storage == "bf16" else torch.float16


def _halfplanes(box, n, seed):
    """n half-planes of a seeded phantom (complex64 [n, box, box/2+1]) and their rotations."""
    fft, rots = synthetic.make_job_torch(box, n, seed, 0.05 if box >= 256 else 0.1, torch.device(DEV),
                                         chunk=max(16, int(1024 * 256 * 256 / (box * box))))
    return fft, torch.from_numpy(rots).to(DEV)


def _quantise(fft, storage):
    """16-bit projections: (stored pairs [n, Y, X, 2], scale [n]), the largest component at 2^14."""
    pairs = torch.view_as_real(fft)
    m = pairs.abs().amax(dim=(1, 2, 3))
    scale = torch.where(m > 0, m / 16384.0, torch.ones_like(m))
    return (pairs * (1.0 / scale)[:, None, None, None]).to(_dtype(storage)), scale


def _images(box, n, seed):
    """n noisy projection images: a soft disc with a gradient under white noise at SNR 0.1."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    u = (torch.arange(box, dtype=torch.float32, device=DEV) - box / 2.0) / (0.3 * box)
    disc = torch.exp(-(u[None, :] ** 2 + u[:, None] ** 2)) * (1.0 + 0.3 * u[None, :])
    img = torch.randn((n, box, box), generator=g, device=DEV)
    return img.mul_(float(disc.std()) / math.sqrt(0.1)).add_(disc)


def _settings(case):
    s = Settings()
    s.SetType(Settings.Type.kFast if case.get("type") == "fast" else Settings.Type.kPrecise)
    s.SetInterpolation(Settings.Interpolation.kDynamic if case.get("interp") == "dynamic"
                       else Settings.Interpolation.kLookup)
    s.SetStorage(STORAGES.index(case["storage"]))
    s.SetAccumulation(Settings.Accumulation.kKahan if case.get("kahan") else Settings.Accumulation.kPlain)
    return s


def _volume(box):
    v = box + 1
    return (torch.zeros((v, v, v), dtype=torch.complex64, device=DEV),
            torch.zeros((v, v, v), dtype=torch.float32, device=DEV))


def _blob_table(settings):
    table = torch.zeros(TABLE, dtype=torch.float32, device=DEV)
    FRB200.FillBlobTable(InputData(None, None, None, None, table), settings)
    return table


def _spaces(rots, box, fast):
    return compute_traverse_spaces(rots, box // 2, box, box, box, fast)


def _counts(text):
    return [int(t) for t in text.split(",")]


def _job_list(text):
    return [tuple(int(v) for v in t.split(":")) for t in text.split(",")]


def _payload(box, n, seed, storage):
    fft, rots = _halfplanes(box, n, seed)
    if storage == "fp32":
        return fft, None, rots
    stored, scale = _quantise(fft, storage)
    return stored, scale, rots


# ---- passes -------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "insert":
        state = _prepare_insert(case, seed)
    elif kind == "jobs":
        state = _prepare_jobs(case, seed)
    elif kind == "serve":
        state = _prepare_serve(case, seed)
    else:
        state = _prepare_prep(case, seed)
    torch.cuda.synchronize()
    state["kind"] = kind
    return state


def _prepare_insert(case, seed):
    box, counts = case["box"], _counts(case["batches"])
    settings = _settings(case)
    fft, scales, rots = _payload(box, sum(counts), seed, case["storage"])
    vol, w = _volume(box)
    table = _blob_table(settings) if case["interp"] == "lookup" else None
    batches, at = [], 0
    for n in counts:
        batches.append((fft[at:at + n], None if scales is None else scales[at:at + n], rots[at:at + n]))
        at += n
    fast = case["type"] == "fast"
    op, out = FRB200(0), OutputData(vol, w)
    big = max(batches, key=lambda b: b[0].shape[0])
    first = InputData(big[0], vol, w, _spaces(big[2], box, fast), table, big[1])
    if not op.Init(out, first, settings):
        raise RuntimeError(op.last_error)
    return {"op": op, "out": out, "first": first, "batches": batches, "table": table, "box": box, "fast": fast}


def _prepare_jobs(case, seed):
    settings = _settings(case)
    jobs = []
    for k, (box, n) in enumerate(_job_list(case["jobs"])):
        fft, scales, rots = _payload(box, n, seed * 1009 + k, case["storage"])
        vol, w = _volume(box)
        jobs.append(InputData(fft, vol, w, _spaces(rots, box, False), None, scales))
    batch = FRBatch(0, torch.cuda.Stream())
    if not batch.Init(settings, len(jobs), sum(int(j.traverse_space.shape[0]) for j in jobs),
                      max(int(j.weight.shape[0]) for j in jobs),
                      sum(bricks_of(int(j.weight.shape[0])) for j in jobs)):
        raise RuntimeError(batch.last_error)
    return {"batch": batch, "jobs": jobs, "table": _blob_table(settings)}


def _prepare_serve(case, seed):
    settings = _settings(case)
    spec = _job_list(case["jobs"])
    jobs = []
    for k, (box, n) in enumerate(spec):
        fft, _, rots = _payload(box, n, seed * 1009 + k, case["storage"])
        jobs.append((box, fft, rots, *_volume(box)))
    side = max(box for box, _ in spec) + 1
    reserve = sum(12 * (box + 1) ** 3 + (4 << 20) for box, _ in spec)
    server = FRServer(0, settings, max_volume_side=side, max_step_projections=8192, max_step_entries=64,
                      staging_bytes=64 << 20, reserve_bytes=reserve)
    return {"server": server, "jobs": jobs, "batch": case["batch"]}


def _prepare_prep(case, seed):
    box, n = case["box"], case["images"]
    p = Prep(box, box, storage=STORAGES.index(case["storage"]), layout=case["layout"])
    dtype = torch.complex64 if case["storage"] == "fp32" else _dtype(case["storage"])
    tail = () if case["storage"] == "fp32" else (2,)
    out = torch.zeros((n, *p.out_shape, *tail), dtype=dtype, device=DEV)
    scales = None if case["storage"] == "fp32" else torch.zeros(n, dtype=torch.float32, device=DEV)
    return {"prep": p, "images": _images(box, n, seed), "out": out, "scales": scales}


def run(state):
    return _RUNS[state["kind"]](state)


def _run_insert(st):
    op, out = st["op"], st["out"]
    out.volume.zero_()
    out.weight.zero_()
    if len(st["batches"]) == 1:  # spaces in hand: the whole reconstruction in one call
        ok = op.Execute(out, st["first"])
    else:
        ok = True
        for fft, scales, rots in st["batches"]:
            spaces = _spaces(rots, st["box"], st["fast"])
            ok = ok and op.Execute(out, InputData(fft, out.volume, out.weight, spaces, st["table"], scales))
    if not ok:
        raise RuntimeError(op.last_error)
    return [out.volume, out.weight]


def _run_jobs(st):
    batch, jobs = st["batch"], st["jobs"]
    batch.stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(batch.stream):
        for j in jobs:
            j.volume.zero_()
            j.weight.zero_()
    if not batch.Execute(jobs, st["table"], graph=True):
        raise RuntimeError(batch.last_error)
    torch.cuda.current_stream().wait_stream(batch.stream)
    return [t for j in jobs for t in (j.volume, j.weight)]


def _run_serve(st):
    server, step = st["server"], st["batch"]
    open_jobs = [server.open_job(box) for box, *_ in st["jobs"]]
    most = max(int(fft.shape[0]) for _, fft, *_ in st["jobs"])
    for at in range(0, most, step):  # the clients' batches arrive interleaved
        for served, (_, fft, rots, _, _) in zip(open_jobs, st["jobs"]):
            if at < fft.shape[0]:
                served.submit(fft[at:at + step], rotations=rots[at:at + step])
    outs = []
    for served in open_jobs:
        served.close()
    for served, (_, _, _, vol, w) in zip(open_jobs, st["jobs"]):
        if served.wait(60.0)["state"] != "done":
            raise RuntimeError("served job failed")
        outs += served.read(vol, w)
        served.release()
    return outs


def _run_prep(st):
    out, scales = st["prep"].Execute(st["images"], st["out"], st["scales"])
    if isinstance(out, BandedPlanes):
        out = out.data
    return [out] if scales is None else [out, scales]


_RUNS = {"insert": _run_insert, "jobs": _run_jobs, "serve": _run_serve, "prep": _run_prep}


# ---- the work a pass cannot do without -------------------------------------------------------

def _insert_work(box, n, storage, fast):
    """A half-plane and a traverse space read per projection; every voxel of its slab rotated and
    tested (25 operations), and per blob pixel (on average 2/3 pi r^2 of a voxel's window) the
    distance, its weight and the complex multiply-add (10)."""
    pixel = 8 if storage == "fp32" else 4
    ball = math.pi * (box / 2 + (0 if fast else RADIUS)) ** 2 / 2
    voxels = ball if fast else (ball + RADIUS * box) * 2 * RADIUS
    flops = voxels * (30 if fast else 25 + 10 * 2 / 3 * math.pi * RADIUS ** 2)
    return n * (pixel * (box // 2 + 1) * box + 112), n * flops


def work(case):
    kind = case["kind"]
    if kind == "prep":
        box, n = case["box"], case["images"]
        pixel = 8 if case["storage"] == "fp32" else 4
        return {"bytes": n * (4 * box * box + pixel * (box // 2 + 1) * box),
                "flops": n * 2.5 * box * box * math.log2(box * box)}
    jobs = [(case["box"], sum(_counts(case["batches"])))] if kind == "insert" else _job_list(case["jobs"])
    nbytes = flops = 0.0
    for box, n in jobs:
        b, f = _insert_work(box, n, case["storage"], case.get("type") == "fast")
        nbytes += b + 12 * (box + 1) ** 3
        flops += f
    return {"bytes": nbytes, "flops": flops}


# ---- the same results in FP64 ---------------------------------------------------------------

def _kaiser(d2):
    """Kaiser-Bessel blob (order 0) at squared distance d2, over its Fourier value at 0."""
    r2 = RADIUS * RADIUS
    i0a = float(torch.special.i0(torch.tensor(ALPHA, dtype=torch.float64)))
    i15 = math.sqrt(2 / (math.pi * ALPHA)) * (math.cosh(ALPHA) - math.sinh(ALPHA) / ALPHA)
    fourier0 = (2 * math.pi) ** 1.5 * RADIUS ** 3 * i15 / (i0a * ALPHA ** 1.5)
    return torch.special.i0(ALPHA * torch.sqrt((1 - d2 / r2).clamp_min(0))) / (i0a * fourier0)


def _insert_exact(box, fft, rots, lookup, fast):
    """The reconstruction of half-planes `fft` (complex128 values taken pixel by pixel) in FP64:
    every voxel of a projection's slab gathers the pixels within the blob radius."""
    v, c = box + 1, box // 2
    nx, ny = box // 2 + 1, box
    vol = torch.zeros(v ** 3, dtype=torch.complex128, device=DEV)
    wgt = torch.zeros(v ** 3, dtype=torch.float64, device=DEV)
    t = rots.double().transpose(1, 2).contiguous()  # image coordinates = t . voxel offset
    axis = t[:, 2, :].abs().argmax(dim=1)
    r = 0.0 if fast else RADIUS
    limit = (box // 2 + r) ** 2
    grid = torch.arange(v, dtype=torch.float64, device=DEV) - c
    table = None
    if lookup:
        table = _kaiser(torch.arange(TABLE, dtype=torch.float64, device=DEV) / (TABLE - 1) * RADIUS ** 2)
    layers = 1 if fast else 8  # 2 r / |normal| <= 2 r sqrt(3) < 7 voxels along the dominant axis
    chunk = max(1, int(1.2e7 / (v * v * layers)))
    for ax in range(3):
        ids = torch.nonzero(axis == ax).flatten()
        ua, va = [(1, 2), (0, 2), (0, 1)][ax]
        for at in range(0, ids.numel(), chunk):
            sel = ids[at:at + chunk]
            tm = t[sel]
            n = tm[:, 2]
            col = -(n[:, ua, None, None] * grid[None, :, None] + n[:, va, None, None] * grid[None, None, :]) / n[:, ax, None, None]
            if fast:
                w = torch.trunc(col + c + 0.5) - c
                w = w[:, None]
                inside = torch.ones_like(w, dtype=torch.bool)
                lo, hi = _columns(tm, box)
                for a, k in ((ua, 2), (va, 3)):
                    shape = [1, 1, 1, 1]
                    shape[k] = v
                    g = (grid + c).view(shape)
                    inside &= (g >= lo[:, a].view(-1, 1, 1, 1)) & (g <= hi[:, a].view(-1, 1, 1, 1))
            else:
                half = (r / n[:, ax].abs())[:, None, None]
                w = torch.ceil(col - half)[:, None] + torch.arange(layers, dtype=torch.float64, device=DEV)[None, :, None, None]
                inside = w <= (col + half)[:, None]
            inside &= (w.abs() <= c) & (w * w + grid[None, None, :, None] ** 2 + grid[None, None, None, :] ** 2 <= limit)
            k, _, iu, iv = torch.nonzero(inside, as_tuple=True)
            p = [None, None, None]
            p[ax], p[ua], p[va] = w[inside], grid[iu], grid[iv]
            q = [tm[k, i, 0] * p[0] + tm[k, i, 1] * p[1] + tm[k, i, 2] * p[2] for i in range(3)]
            voxel = (((p[2] + c) * v + (p[1] + c)) * v + (p[0] + c)).long()
            keep = q[0] >= -r
            if fast:
                x = torch.trunc(q[0] + 0.5).clamp(0, nx - 1).long()
                y = torch.trunc(q[1] + 0.5 + c).clamp(0, ny - 1).long()
                vol.index_add_(0, voxel[keep], _pixels(fft, sel, k[keep], y[keep], x[keep]))
                wgt.index_add_(0, voxel[keep], torch.ones_like(q[0])[keep])
                continue
            k, voxel, qx, qy, z2 = k[keep], voxel[keep], q[0][keep], q[1][keep] + c, q[2][keep] ** 2
            acc = torch.zeros_like(qx, dtype=torch.complex128)
            sw = torch.zeros_like(qx)
            x0, y0 = torch.ceil(qx - r), torch.ceil(qy - r)
            for i in range(4):
                for j in range(4):
                    x, y = x0 + j, y0 + i
                    d2 = (qx - x) ** 2 + (qy - y) ** 2 + z2
                    near = (d2 <= r * r) & (x >= 0) & (x < nx) & (y >= 0) & (y < ny)
                    d2 = torch.where(near, d2, torch.zeros_like(d2))
                    b = table[(d2 * ((TABLE - 1) / (r * r)) + 0.5).long()] if lookup else _kaiser(d2)
                    b = torch.where(near, b, torch.zeros_like(b))
                    px = _pixels(fft, sel, k, y.clamp(0, ny - 1).long(), x.clamp(0, nx - 1).long())
                    acc += b * px
                    sw += b
            vol.index_add_(0, voxel, acc)
            wgt.index_add_(0, voxel, sw)
    return [vol.view(v, v, v), wgt.view(v, v, v)]


def _pixels(fft, sel, k, y, x):
    values, scale = fft
    p = sel[k]
    if scale is None:
        return values[p, y, x].to(torch.complex128)
    pair = values[p, y, x].double() * scale.double()[p, None]
    return torch.complex(pair[:, 0], pair[:, 1])


def _columns(t, box):
    """Integer bounds of the rotated image rectangle [0, B/2] x [-B/2, B/2] in the volume."""
    c = box // 2
    corners = torch.tensor([[c, -c], [c, c], [0, -c], [0, c]], dtype=torch.float64, device=DEV)
    p = torch.einsum("kd,mdj->mkj", corners, t[:, :2, :]) + c
    return torch.floor(p.amin(1).clamp_min(0)), torch.ceil(p.amax(1).clamp_max(box))


def _prep_exact(case, seed):
    box, n = case["box"], case["images"]
    img = _images(box, n, seed)
    nx = box // 2 + 1
    xx, yy = torch.arange(nx, device=DEV)[None, :], torch.arange(box, device=DEV)[:, None]
    factor = (1.0 - 2.0 * ((xx + yy) & 1).double()) / float(box * box)
    stored = case["storage"] != "fp32"
    out, scales = [], []
    for at in range(0, n, 512):
        f = torch.roll(torch.fft.rfft2(img[at:at + 512].double()) * factor, box // 2, dims=1)
        if stored:
            pairs = torch.view_as_real(f)
            scale = pairs.abs().amax(dim=(1, 2, 3)) / 16384.0
            scales.append(scale)
            f = torch.view_as_complex(pairs / scale[:, None, None, None])
        if case["layout"] == "banded":
            stride = 4 * ((nx + 7) // 8 * 8)  # 4-row bands stored column by column, whole 128-byte lines
            flat = torch.zeros((f.shape[0], stride * ((box + 3) // 4)), dtype=f.dtype, device=DEV)
            flat[:, ((yy // 4) * stride + 4 * xx + yy % 4).flatten()] = f.flatten(1)
            f = flat
        out.append(torch.view_as_real(f) if stored else f)
    return [torch.cat(out)] + ([torch.cat(scales)] if stored else [])


def exact(case, seed):
    kind = case["kind"]
    if kind == "prep":
        return _prep_exact(case, seed)
    if kind == "insert":
        specs = [(case["box"], sum(_counts(case["batches"])), seed)]
    else:
        specs = [(box, n, seed * 1009 + k) for k, (box, n) in enumerate(_job_list(case["jobs"]))]
    outs = []
    for box, n, s in specs:
        values, scales, rots = _payload(box, n, s, case["storage"])
        outs += _insert_exact(box, (values, scales), rots, case.get("interp") != "dynamic", case.get("type") == "fast")
    return outs
