"""The performance cases of the sweep-lane library: what its users run, over
the sizes they run it at, through the public entry points of ``espice_b200``.

A case is a dict of plain values; its ``kind`` names the workload:

- ``op``       the operating points of a few lanes with host buffers, from the
               cold start through the ladder: the smallest calls there are;
- ``grid_dc``  independent DC points of the grid-with-diodes deck on the warp
               lanes, device buffers;
- ``analog``   DC points of the 498-unknown BSIM3 analog block at the tight
               setting on the block lanes, FP64 or mixed precision, from the
               nominal operating point: the headline configuration;
- ``mesh``     the uneven batch: eight topologies of 50 to 2,000 unknowns in
               one launch from cold starts, FP64 or mixed precision;
- ``sweep``    sequential .dc sweeps, one per lane, every point returned;
- ``ring``     Monte-Carlo transients of the 31-stage MOS1 ring oscillator on
               the warp lanes;
- ``chain``    Monte-Carlo transients of a BSIM3 inverter chain with streamed
               measure cards on the warp lanes;
- ``digital``  transients of a digital block on a parasitic mesh on the block
               lanes, FP64 or mixed precision;
- ``lu``       the lane refactor + solve alone on a batch of matrices of the
               ring's pattern, the tape compiled into code;
- ``predict``  the learned warm start's inference;
- ``fit``      its training: forward, backward and optimizer steps on the GPU.
"""

import math

import numpy as np
import torch

from espice_b200 import decks, lanes, learned, mlp

TIGHT = dict(reltol=1e-9, vntol=1e-12, abstol=1e-15)
REFINE_SKIP = 1e3


def listed():
    return [
        # one designer's few corners of a small deck: latency alone
        {"name": "op_grid_12", "kind": "op", "lanes": 12},
        # a DC sweep of ordinary length, and a Monte-Carlo batch that fills the GPU
        {"name": "grid_dc_256", "kind": "grid_dc", "lanes": 256},
        {"name": "grid_dc_16411", "kind": "grid_dc", "lanes": 16411},
        # the analog block: an odd batch in FP64, and a large one in mixed precision
        {"name": "analog_fp64_1003", "kind": "analog", "lanes": 1003, "mixed": False},
        {"name": "analog_mixed_12288", "kind": "analog", "lanes": 12288, "mixed": True},
        # many topologies at once
        {"name": "mesh_fp64_96", "kind": "mesh", "lanes": 96, "mixed": False},
        # sequential sweeps of Monte-Carlo samples
        {"name": "sweep_300x101", "kind": "sweep", "lanes": 300, "points": 101},
        # transients: the ring at the configuration's lane count, a measured
        # chain at a corner-analysis count, a block of about 2,000 unknowns
        {"name": "ring_1024", "kind": "ring", "lanes": 1024, "steps": 200},
        {"name": "chain_meas_97", "kind": "chain", "lanes": 97, "stages": 6, "steps": 300},
        {"name": "digital_mixed_148", "kind": "digital", "lanes": 148, "size": 2000, "steps": 6, "mixed": True},
        # the lane LU alone, a batch far larger than L2
        {"name": "lu_ring_131072", "kind": "lu", "lanes": 131072},
        # training the warm start's network (its inference is drawn)
        {"name": "fit_8192", "kind": "fit", "points": 8192, "hidden": 512, "batch": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["op", "grid_dc", "grid_dc", "analog", "analog", "mesh", "sweep", "ring", "chain", "digital",
                       "lu", "predict", "fit"])
    if kind == "op":
        return {"kind": kind, "lanes": _log_int(rng, 1, 200)}
    if kind == "grid_dc":
        return {"kind": kind, "lanes": _log_int(rng, 64, 16384)}
    if kind == "analog":
        mixed = rng.random() < 0.5
        return {"kind": kind, "lanes": _log_int(rng, 100, 8000 if mixed else 4000), "mixed": mixed}
    if kind == "mesh":
        return {"kind": kind, "lanes": _log_int(rng, 16, 256), "mixed": rng.random() < 0.5}
    if kind == "sweep":
        return {"kind": kind, "lanes": _log_int(rng, 16, 300), "points": rng.randint(21, 101)}
    if kind == "ring":
        return {"kind": kind, "lanes": _log_int(rng, 16, 1024), "steps": rng.randint(50, 200)}
    if kind == "chain":
        return {"kind": kind, "lanes": _log_int(rng, 16, 400), "stages": rng.randint(3, 8),
                "steps": rng.randint(50, 300)}
    if kind == "digital":
        return {"kind": kind, "lanes": _log_int(rng, 32, 148), "size": _log_int(rng, 300, 2000),
                "steps": rng.randint(3, 6), "mixed": rng.random() < 0.5}
    if kind == "lu":
        return {"kind": kind, "lanes": 128 * _log_int(rng, 64, 1024)}
    if kind == "predict":
        return {"kind": kind, "lanes": _log_int(rng, 500, 65536), "hidden": rng.choice([128, 256, 512])}
    return {"kind": kind, "points": 256 * rng.randint(8, 32), "hidden": rng.choice([128, 256, 512]),
            "batch": rng.choice([128, 256])}


def _rng(seed):
    return np.random.default_rng(seed)


def _words(n):
    return torch.zeros(n, dtype=torch.int32, device="cuda")


class State:
    """What a program holds across calls: the context and its buffers."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _grid_values(lanes_n, seed):
    fr, slots, values, nominal = decks.grid_diodes_16(seed=seed + 1, points=lanes_n)
    return fr, slots, values, nominal


def _sweep_values(case, seed):
    """Four resistors of the grid scaled per lane, and the swept points."""
    fr, _, _ = decks.grid_diodes(seed=1)
    slots = fr.slots_of(0, "r")[:4]
    nominal = np.array([fr.param(s) for s in slots])
    scales = nominal * np.exp(_rng(seed + 43).uniform(-0.5, 0.5, (case["lanes"], 4)))
    return fr, slots, scales, np.linspace(0.0, 5.0, case["points"])


def _ring_matrices(case, seed):
    """Matrices of the ring's pattern around a diagonally dominant lead, one
    per lane in [entry][lane] planes, and right-hand sides."""
    fr, _, _ = decks.ring_oscillator(lanes=1)
    cp, ri = lanes.pattern(fr)
    lead = _rng(7).uniform(0.5, 2.0, len(ri))
    for j in range(fr.n):
        lead[cp[j] + np.searchsorted(ri[cp[j]:cp[j + 1]], j)] += 8.0
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 17)
    a = torch.rand((len(ri), case["lanes"]), dtype=torch.float64, device="cuda", generator=gen)
    a.mul_(0.2).add_(0.9).mul_(torch.tensor(lead, device="cuda")[:, None])
    rhs = torch.randn((fr.n, case["lanes"]), dtype=torch.float64, device="cuda", generator=gen)
    return fr, cp, ri, lead, a, rhs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "op":
        fr, slots, values, _ = _grid_values(case["lanes"], seed)
        ctx = lanes.DcLanes(fr)
        ctx.set_lanes(slots, values)
        return State(kind=kind, ctx=ctx)
    if kind == "grid_dc":
        fr, slots, values, _ = _grid_values(case["lanes"], seed)
        ctx = lanes.DcLanes(fr)
        ctx.set_lanes(slots, values)
        x = torch.zeros((case["lanes"], fr.n), dtype=torch.float64, device="cuda")
        return State(kind=kind, ctx=ctx, start=torch.zeros_like(x), x=x, it=_words(case["lanes"]),
                     st=_words(case["lanes"]), opts=lanes.newton_opts())
    if kind == "analog":
        fr, expand = decks.analog_block()
        params, nominal = decks.analog_block_params(seed=seed + 1, points=case["lanes"])
        opts = lanes.newton_opts(**TIGHT)
        ctx = lanes.DcLanes(fr)
        ctx.set_mode(precision=lanes.PREC_FP64, path=lanes.PATH_BLOCK)
        ctx.set_lanes(expand.slots, expand(nominal))
        x_nominal = ctx.solve(x0=None, opts=opts)[0][0]
        if case["mixed"]:
            ctx.set_mode(precision=lanes.PREC_MIXED, path=lanes.PATH_BLOCK, refine_skip=REFINE_SKIP)
        ctx.set_lanes(expand.slots, expand.lane_params(params), cols=expand.cols)
        start = torch.tensor(x_nominal, device="cuda").repeat(case["lanes"], 1)
        return State(kind=kind, ctx=ctx, start=start, x=torch.empty_like(start), it=_words(case["lanes"]),
                     st=_words(case["lanes"]), opts=opts)
    if kind == "mesh":
        rng = _rng(seed + 31)
        ctxs, xs, its, sts = [], [], [], []
        for size in decks.MESH_GATES_SIZES:
            fr, slots = decks.mesh_gates(size)
            c = lanes.DcLanes(fr)
            c.set_mode(precision=lanes.PREC_MIXED if case["mixed"] else lanes.PREC_FP64, path=lanes.PATH_BLOCK,
                       refine_skip=REFINE_SKIP if case["mixed"] else 0.0)
            c.set_lanes(slots, rng.uniform(0.8, 1.8, (case["lanes"], 1)))
            ctxs.append(c)
            xs.append(torch.zeros((case["lanes"], fr.n), dtype=torch.float64, device="cuda"))
            its.append(_words(case["lanes"]))
            sts.append(_words(case["lanes"]))
        return State(kind=kind, ctxs=ctxs, xs=xs, its=its, sts=sts)
    if kind == "sweep":
        fr, slots, scales, points = _sweep_values(case, seed)
        ctx = lanes.DcLanes(fr)
        ctx.set_lanes(slots, scales)
        return State(kind=kind, ctx=ctx, slot=fr.slot("vin", "dc"), values=points)
    if kind == "ring":
        fr, slots, values = decks.ring_oscillator(seed=seed + 1, lanes=case["lanes"])
        ctx = lanes.DcLanes(fr)
        ctx.set_lanes(slots, values)
        return State(kind=kind, ctx=ctx,
                     opts=lanes.tran_opts(case["steps"] * decks.RING_T_STEP, decks.RING_T_STEP, decks.RING_T_MAX),
                     x=torch.zeros((case["lanes"], fr.n), dtype=torch.float64, device="cuda"),
                     stats=torch.zeros((case["lanes"], len(lanes.TS_FIELDS)), dtype=torch.int32, device="cuda"))
    if kind == "chain":
        t_step = 5e-12
        t_stop = case["steps"] * t_step
        fr, slots, values = decks.bsim3_inverters(
            seed=seed + 1, stages=case["stages"], lanes=case["lanes"], c_load=10e-15,
            pulse=[0.0, 1.8, 0.1 * t_stop, 50e-12, 50e-12, 0.4 * t_stop, 2.0 * t_stop])
        ctx = lanes.DcLanes(fr)
        ctx.set_lanes(slots[1:], values[:, 1:])
        first, last = fr.unknown("s0"), fr.unknown(f"s{case['stages'] - 1}")
        meas = [lanes.when(first, 0.9, fall=1), lanes.when(last, 0.9, cross=1),
                lanes.window(lanes.MEAS_MAX, last), lanes.window(lanes.MEAS_AVG, first)]
        return State(kind=kind, ctx=ctx, meas=meas, opts=lanes.tran_opts(t_stop, t_step, t_step))
    if kind == "digital":
        t_step = 10e-12
        fr, slots = decks.digital_block(size=case["size"], n_cells=max(4, case["size"] // 40), n_inputs=8)
        ctx = lanes.DcLanes(fr)
        ctx.set_mode(precision=lanes.PREC_MIXED if case["mixed"] else lanes.PREC_FP64, path=lanes.PATH_BLOCK,
                     refine_skip=REFINE_SKIP if case["mixed"] else 0.0)
        ctx.set_lanes(slots, decks.digital_block_vto(len(slots), case["lanes"], seed=seed + 3))
        return State(kind=kind, ctx=ctx, opts=lanes.tran_opts(case["steps"] * t_step, t_step, t_step),
                     x=torch.zeros((case["lanes"], fr.n), dtype=torch.float64, device="cuda"),
                     stats=torch.zeros((case["lanes"], len(lanes.TS_FIELDS)), dtype=torch.int32, device="cuda"))
    if kind == "lu":
        fr, _, _, lead, a, rhs = _ring_matrices(case, seed)
        ctx = lanes.DcLanes(fr)
        dx = torch.zeros_like(rhs)
        bad = torch.zeros(case["lanes"], dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        # a program builds the tape's kernel once, on a small batch
        ctx.lu_lanes_compiled(lead, a[:, :32].contiguous().data_ptr(), rhs[:, :32].contiguous().data_ptr(),
                              torch.zeros_like(rhs[:, :32]).contiguous().data_ptr(), bad.data_ptr(), 32)
        return State(kind=kind, ctx=ctx, lead=lead, a=a, rhs=rhs, dx=dx, bad=bad)
    if kind == "predict":
        net = mlp.Mlp(16, case["hidden"], 3, 498, seed=seed + 1)
        x = torch.tensor(_rng(seed + 5).standard_normal((case["lanes"], 16)), dtype=torch.float32, device="cuda")
        y = torch.zeros((case["lanes"], 498), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return State(kind=kind, net=net, x=x, y=y)
    # fit: smooth targets of the points' parameters, as operating points are
    rng = _rng(seed + 6)
    params, _ = decks.analog_block_params(seed=seed + 1, points=case["points"])
    z = (params - params.mean(0)) / params.std(0)
    y = np.tanh(z @ rng.normal(0.0, 0.25, (16, 498))) + 0.1 * (z @ rng.normal(0.0, 0.25, (16, 498)))
    return State(kind=kind, params=params, targets=y, hidden=case["hidden"], batch=case["batch"], seed=seed + 1)


def run(s):
    if s.kind == "op":
        x, it, st, rung, _ = s.ctx.op()
        return {"x": x, "iters": it, "status": st, "rung": rung}
    if s.kind in ("grid_dc", "analog"):
        s.x.copy_(s.start)
        torch.cuda.current_stream().synchronize()  # the library's stream reads the starts
        s.ctx.solve_device(s.x.data_ptr(), s.it.data_ptr(), s.st.data_ptr(), opts=s.opts)
        return {"x": s.x, "iters": s.it, "status": s.st}
    if s.kind == "mesh":
        lanes.group_solve_device(s.ctxs, [x.data_ptr() for x in s.xs], [w.data_ptr() for w in s.its],
                                 [w.data_ptr() for w in s.sts], cold=[True] * len(s.ctxs))
        return {"x": s.xs, "iters": s.its, "status": s.sts}
    if s.kind == "sweep":
        x, it, cv, st, _ = s.ctx.sweep(s.slot, s.values)
        return {"x": x, "iters": it, "converged": cv, "status": st}
    if s.kind in ("ring", "digital"):
        s.ctx.tran_device(s.opts, s.x.data_ptr(), s.stats.data_ptr())
        return {"x": s.x, "stats": s.stats}
    if s.kind == "chain":
        v, st, x, _ = s.ctx.tran_meas(s.opts, s.meas)
        return {"measures": v, "stats": st, "x": x}
    if s.kind == "lu":
        s.ctx.lu_lanes_compiled(s.lead, s.a.data_ptr(), s.rhs.data_ptr(), s.dx.data_ptr(), s.bad.data_ptr(),
                                s.a.shape[1])
        return {"dx": s.dx, "bad": s.bad}
    if s.kind == "predict":
        s.net.predict(s.x.data_ptr(), s.x.shape[0], s.y.data_ptr())
        return s.y
    ws = learned.LearnedWarmStart(16, 498, hidden=s.hidden, layers=3, seed=s.seed)
    loss = ws.fit(s.params, s.targets, epochs=2, batch=s.batch, lr=1e-3, lr_end=1e-3, seed=s.seed)
    weights = [w for layer in ws.net.weights() for w in layer]
    ws.close()
    return {"loss": loss, "weights": weights}


# Unknowns, live values a lane, matrix-factor multiply-subtracts and model
# instances of the fixed decks, for the work counts below.
_GRID = dict(n=82, live=16, flops=2.0e3)
_ANALOG = dict(n=498, live=16, flops=1.6e5)
_MESH_FLOPS = {50: 1e3, 100: 3e3, 200: 1e4, 400: 3e4, 700: 8e4, 1000: 1.5e5, 1500: 3e5, 2000: 5e5}


def work(case):
    """Inputs once (the lanes' live parameter values, their starts) and
    outputs once; the multiply-subtracts of two Newton iterations' factors
    (the least the gates allow) per solve or time step."""
    kind, n_l = case["kind"], case.get("lanes", 0)
    if kind in ("op", "grid_dc"):
        return {"bytes": n_l * 8.0 * (2 * _GRID["n"] + _GRID["live"] + 1), "flops": n_l * 2 * 2 * _GRID["flops"]}
    if kind == "analog":
        return {"bytes": n_l * 8.0 * (2 * _ANALOG["n"] + _ANALOG["live"] + 1),
                "flops": n_l * 2 * 2 * _ANALOG["flops"]}
    if kind == "mesh":
        return {"bytes": n_l * 8.0 * sum(s + 2 for s in decks.MESH_GATES_SIZES),
                "flops": n_l * 4 * sum(_MESH_FLOPS.values())}
    if kind == "sweep":
        return {"bytes": n_l * (32.0 + case["points"] * (8.0 * _GRID["n"] + 5)),
                "flops": n_l * case["points"] * 4 * _GRID["flops"]}
    if kind == "ring":
        return {"bytes": n_l * (8.0 * (62 + 34) + 32), "flops": n_l * case["steps"] * 4 * 300.0}
    if kind == "chain":
        return {"bytes": n_l * 8.0 * (4 * case["stages"] + 12), "flops": n_l * case["steps"] * 4 * 20.0 * case["stages"]}
    if kind == "digital":
        return {"bytes": n_l * 8.0 * (1.1 * case["size"] + 4), "flops": n_l * case["steps"] * 4 * 250.0 * case["size"]}
    if kind == "lu":
        # the ring's pattern: 34 unknowns, 129 entries
        return {"bytes": n_l * (8.0 * (129 + 2 * 34) + 1), "flops": n_l * 2 * 500.0}
    h = case["hidden"]
    w = 16 * h + h * h + h * 498
    if kind == "predict":
        return {"bytes": n_l * 4.0 * (16 + 498) + 2.0 * w, "flops": 2.0 * n_l * w}
    return {"bytes": 2 * case["points"] * 4.0 * (16 + 498) + 8.0 * w, "flops": 2 * 6.0 * case["points"] * w}


def _grid_exact(fr, slots, values):
    """Every lane's DC solution of the grid-with-diodes deck by a damped
    Newton iteration on its own equations, batched over the lanes."""
    if len(values) > 4096:
        return np.concatenate([_grid_exact(fr, slots, values[k:k + 4096]) for k in range(0, len(values), 4096)])
    n, m = fr.n, values.shape[0]
    tables = {t: (np.asarray(nd).astype(np.int64), np.asarray(p, np.float64)) for t, nd, p in fr.batches}
    col = {(fr.batches[s.batch][0], s.inst, s.param): c for c, s in enumerate(slots)}
    vals = torch.tensor(values, dtype=torch.float64, device="cuda")
    lin = torch.zeros((m, n, n), dtype=torch.float64, device="cuda")
    rhs = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    lin[:, 0, 0] = 1.0
    nd, p = tables[0]
    for k, (i, j) in enumerate(nd):
        g = 1.0 / vals[:, col[(0, k, 0)]] if (0, k, 0) in col else 1.0 / p[k, 0]
        for r, c, sgn in ((i, i, 1), (j, j, 1), (i, j, -1), (j, i, -1)):
            lin[:, r, c] += sgn * g
    nd, p = tables[2]
    for k, (i, j, b) in enumerate(nd):
        for r, c, sgn in ((i, b, 1), (j, b, -1), (b, i, 1), (b, j, -1)):
            lin[:, r, c] += sgn
        rhs[:, b] = vals[:, col[(2, k, 0)]] if (2, k, 0) in col else p[k, 0]
    nd, p = tables[4]
    a, c, ai = nd.T
    is_, rs, gmin = (torch.tensor(p[:, k], device="cuda") for k in (0, 2, 11))
    vt = 1.380649e-23 * 300.15 / 1.602176634e-19
    for k in range(len(a)):
        for r, q, sgn in ((a[k], a[k], 1), (ai[k], ai[k], 1), (a[k], ai[k], -1), (ai[k], a[k], -1)):
            lin[:, r, q] += sgn / rs[k]
    x = torch.zeros_like(rhs)
    vd = torch.zeros((m, len(a)), dtype=torch.float64, device="cuda")
    for _ in range(200):
        e = torch.exp(vd.clamp(max=3.0) / vt)
        cur, g = is_ * (e - 1.0) + gmin * vd, is_ / vt * e + gmin
        ieq = cur - g * vd
        jac, b = lin.clone(), rhs.clone()
        for k in range(len(a)):
            for r, q, sgn in ((ai[k], ai[k], 1), (c[k], c[k], 1), (ai[k], c[k], -1), (c[k], ai[k], -1)):
                jac[:, r, q] += sgn * g[:, k]
            b[:, ai[k]] -= ieq[:, k]
            b[:, c[k]] += ieq[:, k]
        jac[:, 0, :] = 0.0
        jac[:, 0, 0] = 1.0
        b[:, 0] = 0.0
        x = torch.linalg.solve(jac, b.unsqueeze(2))[:, :, 0]
        new = x[:, ai] - x[:, c]
        up = torch.where(vd > 0.4, vd + vt * torch.log1p((new - vd).clamp(min=0.0) / vt), new.clamp(max=0.6))
        step = torch.where(new > vd, up, new) - vd
        vd = vd + step
        if float(step.abs().max()) < 1e-13:
            break
    return x.cpu().numpy()


def exact(case, seed):
    """The outputs that follow from the inputs alone, in 64 bits: the DC
    points of the diode deck, the linear solves and the network's inference.
    The MOSFET models and the training run have no plain form here."""
    kind = case["kind"]
    if kind in ("op", "grid_dc"):
        fr, slots, values, _ = _grid_values(case["lanes"], seed)
        x = _grid_exact(fr, slots, values)
        if kind == "op":
            return {"x": x, "iters": None, "status": None, "rung": None}
        return {"x": x, "iters": None, "status": None}
    if kind == "sweep":
        fr, slots, scales, points = _sweep_values(case, seed)
        lane_values = np.repeat(scales, len(points), axis=0)
        swept = np.tile(points, len(scales))[:, None]
        x = _grid_exact(fr, slots + [fr.slot("vin", "dc")], np.hstack([lane_values, swept]))
        return {"x": x.reshape(len(scales), len(points), fr.n), "iters": None, "converged": None, "status": None}
    if kind == "lu":
        fr, cp, ri, _, a, rhs = _ring_matrices(case, seed)
        cols = np.repeat(np.arange(fr.n), np.diff(cp.astype(np.int64)))
        out = torch.empty_like(rhs)
        for k in range(0, case["lanes"], 8192):
            sl = slice(k, min(k + 8192, case["lanes"]))
            dense = torch.zeros((sl.stop - sl.start, fr.n, fr.n), dtype=torch.float64, device="cuda")
            dense[:, ri.astype(np.int64), cols] = a[:, sl].T
            out[:, sl] = torch.linalg.solve(dense, -rhs[:, sl].T.unsqueeze(2))[:, :, 0].T
        return {"dx": out, "bad": None}
    if kind == "predict":
        s = prepare(case, seed)
        h = s.x.double()
        layers = s.net.weights()
        for i, (w, b) in enumerate(layers):
            w, b = torch.tensor(w, device="cuda").double(), torch.tensor(b, device="cuda").double()
            h = torch.nn.functional.pad(h, (0, w.shape[1] - h.shape[1])) @ w.T + b
            if i + 1 < len(layers):
                h = torch.tanh(h)
        return h[:, :498]
    return None
