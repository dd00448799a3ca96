"""Timed cases of the framework's public entry points.

A case names one call path (`op`), a field (generator, dimensions, type) and
the options of the call:

* compress    Compressor.compress_pipeline on a device-resident field
* decompress  Compressor.decompress_pipeline of a device-resident container
* retrieve    Compressor.progressive: open, one step per target, plane state
* batch       Batch.compress of many uneven fields (one launch per stage)
* report      Handle.statistics of a reconstruction against its original
* serve       Server: a burst of retrievals over several resident fields

Sizes, bounds and field families are those of bench.py, the tests and
prism_b200.fields (128^3 float, 384x384x256 double, 1024^3 float, the uneven
mix), plus ragged and low-dimensional shapes of the same ranges.

Containers, reconstructions and plane states are defined bit for bit by the
container format (explicitly rounded arithmetic), so they must stay the same;
the statistics' squared-error sum and the server's refinement sums depend on
the order of additions and carry a tolerance.
"""
import math

import numpy as np
import torch

import prism_b200 as P
from prism_b200 import fields

F32, F64 = "float32", "float64"


def listed():
    return [
        # smallest call: a small block of a simulation, bounded by launches and waits
        dict(name="compress-64x48x40-f32", op="compress", kind="sinusoid", nx=64, ny=48, nz=40, dtype=F32, rel=True,
             bound=1e-3, prog=False),
        # ordinary snapshot of a smooth variable (8 MB), one way and back
        dict(name="compress-128-f32", op="compress", kind="sinusoid", nx=128, ny=128, nz=128, dtype=F32, rel=True,
             bound=1e-4, prog=False),
        dict(name="decompress-128-f32", op="decompress", kind="sinusoid", nx=128, ny=128, nz=128, dtype=F32, rel=True,
             bound=1e-4),
        # a 2-D slice or surface field with odd extents
        dict(name="compress-1799x901-f32", op="compress", kind="grf", nx=1799, ny=901, nz=1, dtype=F32, rel=True,
             bound=1e-4, prog=False),
        # double-precision turbulence variable stored for progressive use, then
        # retrieved at five bounds, each step refining the previous one
        dict(name="compress-384x384x256-f64-prog", op="compress", kind="grf", nx=384, ny=384, nz=256, dtype=F64,
             rel=True, bound=1e-6, prog=True),
        dict(name="retrieve-384x384x256-f64-chain", op="retrieve", kind="grf", nx=384, ny=384, nz=256, dtype=F64,
             rel=True, bound=1e-6, targets="1e-2 1e-3 1e-4 1e-5 1e-6", exact=False),
        # one coarse look at a small ragged field (latency of a single retrieval)
        dict(name="retrieve-100x90x77-f32", op="retrieve", kind="sparse", nx=100, ny=90, nz=77, dtype=F32, rel=True,
             bound=1e-5, targets="1e-3", exact=False),
        # largest: a sparse, sharp 4.3 GB field at an absolute bound
        dict(name="compress-1024-f32-sparse", op="compress", kind="sparse", nx=1024, ny=1024, nz=1024, dtype=F32,
             rel=False, bound=1e-3, prog=False),
        # large ragged field on the way back
        dict(name="decompress-1000x777x513-f32-sparse", op="decompress", kind="sparse", nx=1000, ny=777, nz=513,
             dtype=F32, rel=False, bound=1e-3),
        # many variables and blocks of uneven shapes at once (1-D, 2-D, 3-D)
        dict(name="batch-32-uneven-f32", op="batch", count=32, mix=47, cap=256, dtype=F32, rel=True, bound=1e-3,
             prog=False),
        # quality report of a reconstruction
        dict(name="report-384x384x256-f64", op="report", kind="grf", nx=384, ny=384, nz=256, dtype=F64, rel=True,
             bound=1e-6),
        # retrieval service: a burst of requests over resident fields with room
        # for a few reconstructions only
        dict(name="serve-6-fields-f64", op="serve", kind="grf", count=6, nx=150, ny=150, nz=96, dtype=F64, rel=True,
             bound=1e-6, requests=24, slots=4, room=4.2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["compress"] * 4 + ["decompress"] * 3 + ["retrieve"] * 3 + ["batch", "report", "serve"])
    dtype = rng.choice([F32, F32, F64])
    rel = rng.random() < 0.7
    c = dict(op=op, dtype=dtype, rel=rel, bound=float("%.3g" % _log(rng, 1e-6 if dtype == F64 else 1e-5, 1e-2)))
    if op == "batch":
        c.update(count=rng.randint(3, 48), mix=rng.randint(0, 10 ** 6), cap=rng.choice([96, 160, 224]),
                 prog=rng.random() < 0.3)
        return c
    c["kind"] = rng.choice(["sinusoid", "grf", "sparse"])
    if op == "serve":
        e = int(_log(rng, 40, 170))
        c.update(count=rng.randint(2, 8), nx=e + rng.randint(0, 20), ny=e + rng.randint(0, 20),
                 nz=max(8, e - rng.randint(0, 20)), requests=rng.randint(8, 40), slots=rng.randint(2, 8),
                 room=round(rng.uniform(2.2, 6.0), 1), rel=True, bound=min(c["bound"], 1e-4))
        return c
    d = rng.random()
    if d < 0.72:  # 3-D, up to 2^28 float or 2^27 double values (1 GB)
        n = _log(rng, 2e4, (2 ** 28 if dtype == F32 else 2 ** 27) / (2 if op == "retrieve" else 1))
        a, b = _log(rng, 0.5, 2.0), _log(rng, 0.5, 2.0)
        e = (n / (a * b)) ** (1 / 3)
        nx, ny, nz = max(8, int(e * a)), max(8, int(e * b)), max(8, int(e))
    elif d < 0.92:  # 2-D
        nx, ny, nz = int(_log(rng, 64, 4096)), int(_log(rng, 64, 4096)), 1
    else:  # 1-D
        nx, ny, nz = int(_log(rng, 512, 2 ** 20)), 1, 1
    c.update(nx=nx, ny=ny, nz=nz)
    if op == "compress":
        c["prog"] = rng.random() < 0.4
    if op == "retrieve":
        c.update(bound=min(c["bound"], 1e-4), exact=rng.random() < 0.3)
        scale = 1.0 if rel else 1e-1
        steps = sorted((_log(rng, c["bound"], 1e-1) for _ in range(rng.randint(1, 5))), reverse=True)
        c["targets"] = " ".join("%.3g" % (t * scale) for t in steps)
    return c


def _dtype(case):
    return np.dtype(case["dtype"])


def _sparse(shape, dtype, seed, cells=64, zero_frac=0.3, spike_frac=1e-3, spike_amp=1e3):
    """Piecewise-quadratic cells, 30% of them exactly zero, and 0.1% isolated
    spikes: fields.device_voronoi with the nearest seed found per block of 8
    values along each axis, so that multi-GB fields take a fraction of a second."""
    nz, ny, nx = shape
    rng = np.random.default_rng(seed)
    ext = [(nz + 7) // 8, (ny + 7) // 8, (nx + 7) // 8]
    seeds = rng.uniform(0.0, 1.0, (cells, 3)) * np.array(ext)
    coef = rng.normal(0.0, 1.0, (cells, 10))
    coef[rng.uniform(0.0, 1.0, cells) < zero_frac] = 0.0
    coef = torch.tensor(coef, device="cuda", dtype=torch.float32)
    ax = [torch.arange(e, device="cuda", dtype=torch.float32) for e in ext]
    best = owner = None
    for c in range(cells):
        d = ((ax[0] - float(seeds[c, 0])) ** 2)[:, None, None] + ((ax[1] - float(seeds[c, 1])) ** 2)[:, None] \
            + (ax[2] - float(seeds[c, 2])) ** 2
        if best is None:
            best, owner = d, torch.zeros(ext, device="cuda", dtype=torch.long)
        else:
            owner = torch.where(d < best, c, owner)
            best = torch.minimum(d, best)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    out = torch.empty(shape, device="cuda", dtype=tdt)
    y = (torch.arange(ny, device="cuda", dtype=torch.float32) / ny)[:, None]
    x = torch.arange(nx, device="cuda", dtype=torch.float32) / nx
    iy, ix = torch.arange(ny, device="cuda") // 8, torch.arange(nx, device="cuda") // 8
    for bz in range(ext[0]):
        o = owner[bz][iy][:, ix]
        k = [coef[:, i][o] for i in range(10)]
        flat = k[0] + k[1] * x + k[2] * y + k[4] * x * x + k[5] * y * y + k[7] * x * y
        lin, quad = k[3] + k[8] * y + k[9] * x, k[6]
        z0, z1 = 8 * bz, min(nz, 8 * bz + 8)
        z = (torch.arange(z0, z1, device="cuda", dtype=torch.float32) / nz)[:, None, None]
        out[z0:z1] = (flat + lin * z + quad * z * z).to(tdt)
    n = out.numel()
    spikes = int(round(n * spike_frac))
    if spikes:
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        at = torch.unique(torch.randint(0, n, (spikes,), device="cuda", generator=g))
        sign = torch.where(torch.rand(at.numel(), device="cuda", generator=g) < 0.5, -1.0, 1.0)
        out.view(-1)[at] = (sign * spike_amp).to(tdt)
    return out


def _field(kind, shape, dtype, seed):
    gen = {"sinusoid": fields.device_sinusoid, "grf": fields.device_grf, "sparse": _sparse}[kind]
    return gen(tuple(shape), dtype, seed).contiguous()


def _context(case, prog):
    return P.Context(case["nx"], case["ny"], case["nz"], _dtype(case), P.REL if case["rel"] else P.ABS,
                     case["bound"], prog)


def _targets(case):
    return [float(t) for t in case["targets"].split()]


def _prepare_serve(case, seed):
    ctx = _context(case, True)
    comp = P.Compressor(ctx)
    conts = [comp.compress_pipeline(_field(case["kind"], ctx.shape, ctx.dtype, seed + 97 * i)).clone()
             for i in range(case["count"])]
    rng = np.random.default_rng(seed)
    reqs = [(int(rng.integers(case["count"])), float(np.exp(rng.uniform(np.log(case["bound"]), np.log(1e-1)))))
            for _ in range(case["requests"])]
    probe = P.Server(1 << 40, slots=case["slots"])
    for k in conts:
        probe.add_field(ctx, k)
    st = probe.stats()
    probe.close()
    value_bytes = case["nx"] * case["ny"] * case["nz"] * ctx.tsize
    # every slot can hold the entry it computes and the one it refines
    room = max(case["room"], 2.0 * case["slots"] + 0.2)
    server = P.Server(int(st["bytes_resident"] + st["bytes_reserved"] + room * value_bytes), slots=case["slots"])
    ids = [server.add_field(ctx, k) for k in conts]
    tdt = torch.float32 if case["dtype"] == F32 else torch.float64
    outs = [torch.empty(ctx.shape, dtype=tdt, device="cuda") for _ in reqs]
    comp.h.close()
    return dict(op="serve", server=server, reqs=[(ids[f], t) for f, t in reqs], outs=outs)


def prepare(case, seed):
    op, dt = case["op"], _dtype(case)
    if op == "batch":
        items = []
        for i, (kind, (nx, ny, nz)) in enumerate(fields.uneven_mix(case["count"], case["mix"], cap3=case["cap"] ** 3)):
            ctx = P.Context(nx, ny, nz, dt, P.REL if case["rel"] else P.ABS, case["bound"], case["prog"])
            items.append((ctx, _field(kind, ctx.shape, dt, seed + i)))
        batch = P.Batch(items)
        for out in batch.outs:  # the containers' sizes vary: the buffers are compared whole
            out.zero_()
        return dict(op=op, batch=batch)
    if op == "serve":
        return _prepare_serve(case, seed)
    ctx = _context(case, case.get("prog", op == "retrieve"))
    data = _field(case["kind"], ctx.shape, dt, seed)
    if op == "report":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 1)
        noise = torch.rand(ctx.shape, dtype=data.dtype, device="cuda", generator=g) - 0.5
        eb = case["bound"] * (float(data.max() - data.min()) if case["rel"] else 1.0)
        return dict(op=op, handle=P.Handle(), data=data, rec=data + noise * (2.0 * eb))
    comp = P.Compressor(ctx)
    if op == "compress":
        return dict(op=op, comp=comp, data=data,
                    out=torch.zeros(comp.max_container_size(), dtype=torch.uint8, device="cuda"))
    cont = comp.compress_pipeline(data).clone()
    if op == "decompress":
        return dict(op=op, comp=comp, cont=cont, out=torch.empty_like(data))
    return dict(op=op, comp=comp, cont=cont, targets=_targets(case), exact=case["exact"])


def run(state):
    op = state["op"]
    if op == "compress":
        cont = state["comp"].compress_pipeline(state["data"], state["out"])
        return dict(container=state["out"], size=cont.numel())
    if op == "decompress":
        return state["comp"].decompress_pipeline(state["cont"], state["out"])
    if op == "retrieve":
        prog = state["comp"].progressive(state["cont"])
        if state["exact"]:
            prog.exact()
        for target in state["targets"]:
            values = prog.step(target)
        begin, end, maxlevel = prog.state()
        prog.close()
        return dict(values=values, begin=begin, end=end, maxlevel=maxlevel)
    if op == "batch":
        conts, _ = state["batch"].compress()
        return dict(containers=state["batch"].outs, sizes=np.array([c.numel() for c in conts]))
    if op == "report":
        return state["handle"].statistics(state["data"], state["rec"])
    server = state["server"]
    ids = [server.submit(f, t, out) for (f, t), out in zip(state["reqs"], state["outs"])]
    for i in ids:
        server.wait(i)
    return state["outs"]


def _mix_values(case):
    return sum(nx * ny * nz for _, (nx, ny, nz) in
               fields.uneven_mix(case["count"], case["mix"], cap3=case["cap"] ** 3))


def work(case):
    """Field and container each moved once (the container taken as a quarter of
    the field, near the measured ratios at these bounds); a refinement step
    reads the previous values and writes the new ones; about a dozen
    operations of the spline predictor and quantiser per value."""
    op, size = case["op"], _dtype(case).itemsize
    n = _mix_values(case) if op == "batch" else case["nx"] * case["ny"] * case["nz"]
    field, cont = n * size, n * size / 4
    if op == "report":
        return {"bytes": 2 * field, "flops": 6 * n}
    if op == "serve":
        return {"bytes": case["requests"] * field, "flops": 12 * n * case["requests"]}
    if op == "retrieve":
        steps = len(_targets(case))
        return {"bytes": cont + field * (2 * steps - 1), "flops": 12 * n * steps}
    return {"bytes": field + cont, "flops": 12 * n}


def tolerance(case):
    if case["op"] == "report":  # a sum of n squares in double, in some order
        return {"rel": 1e-11, "max": 1e-11}
    if case["op"] == "serve":
        # a result is one step, or the sum of a resident coarser result and a
        # refinement: a few roundings apart, per step of the chain
        eps = float(np.finfo(_dtype(case)).eps)
        return {"rel": 16 * eps, "max": 64 * eps}
    return "exact"


def exact(case, seed):
    """64-bit values for the report.  Containers and retrieved values are
    defined by the format's own rounding, bit for bit, and compared exactly."""
    if case["op"] != "report":
        return None
    state = prepare(case, seed)
    data, rec = state["data"].double().reshape(-1), state["rec"].double().reshape(-1)
    err = (rec - data).abs()
    lo, hi = float(data.min()), float(data.max())
    l2, worst = float((err * err).sum()), float(err.max())
    mse = l2 / data.numel()
    return dict(max_err=worst, max_rel_err=worst / (hi - lo), psnr=20 * math.log10(hi - lo) - 10 * math.log10(mse),
                nrmse=math.sqrt(mse) / (hi - lo), min=lo, max=hi, l2=l2, max_err_index=None)
