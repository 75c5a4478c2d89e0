"""The task programs at the edges of their forms (B200): one warp's stream, a
CTA's of 256 and of 128 threads, compact and wide words, shared memory and
the slab. Every form runs the same operations in the same order, so the
lanes agree bit for bit.

- A lane of a batch large enough for the narrow CTAs equals the same lane of
  a small batch (wide CTAs), FP64 and mixed.
- FP64 block lanes equal the warp lanes (the largest ones' words streamed).
- A value space past the compact words' 65,536 equals the oracle.
- Training: a step replayed as a graph equals one launched by itself.
"""

import numpy as np
import pytest

from espice_b200 import decks, lanes, mlp
from espice_b200.circuit import Circuit
from oracle import oracle

pytestmark = pytest.mark.gpu


def ladder(sections):
    """A resistor ladder with a diode at its end: sections + 3 unknowns."""
    c = Circuit()
    c.V("vin", "n0", "0", dc=1.0)
    for k in range(sections):
        c.R(f"r{k}", f"n{k}", f"n{k + 1}", 100.0 + k)
        c.R(f"g{k}", f"n{k + 1}", "0", 1e4)
    c.D("d0", f"n{sections}", "0", is_=1e-14, n=1.0, rs=10.0)
    fr = c.freeze()
    return fr, [fr.slot("vin", "dc")], lambda n: np.linspace(0.5, 3.0, n).reshape(-1, 1)


def mesh(size):
    fr, slots = decks.mesh_gates(size)
    return fr, slots, lambda n: np.linspace(0.8, 1.8, n).reshape(-1, 1)


def grid(_):
    fr, slots, _ = decks.grid_diodes(seed=1)
    return fr, slots, lambda n: np.linspace(0.0, 5.0, n).reshape(-1, 1)


def solve(fr, slots, values, precision, path):
    ctx = lanes.DcLanes(fr)
    ctx.set_mode(precision=precision, path=path)
    ctx.set_lanes(slots, values)
    x, it, st, stats = ctx.solve(x0=np.zeros(fr.n))
    ctx.close()
    return x.view(np.uint64), it, st


def width(fr, slots, values, precision):
    """Threads of the CTAs these lanes run best on."""
    ctx = lanes.DcLanes(fr)
    ctx.set_mode(precision=precision, path=lanes.PATH_BLOCK)
    ctx.set_lanes(slots, values[:1])
    ctx.solve(x0=np.zeros(fr.n))
    ctx.set_lanes(slots, values)
    w = ctx.block_info()["width"]
    ctx.close()
    return w


@pytest.mark.parametrize("precision", [lanes.PREC_FP64, lanes.PREC_MIXED])
@pytest.mark.parametrize("deck,size", [(ladder, 1), (ladder, 31), (ladder, 130), (grid, 0), (mesh, 50), (mesh, 200),
                                       (mesh, 400)])
def test_narrow_ctas_equal_wide(deck, size, precision):
    fr, slots, values = deck(size)
    # 1,200 lanes: more than any form holds at once on wide CTAs
    big = values(1200)
    pick = np.r_[0:3, 593:596, 1197:1200]
    a = solve(fr, slots, big, precision, lanes.PATH_BLOCK)
    b = solve(fr, slots, big[pick], precision, lanes.PATH_BLOCK)
    for u, v in zip(a, b):
        assert np.array_equal(u[pick], v)
    # (four narrow FP64 lanes of the 400-unknown mesh would lie in global memory: it stays wide)
    narrow = 256 if (deck, size, precision) == (mesh, 400, lanes.PREC_FP64) else 128
    assert (width(fr, slots, big, precision), width(fr, slots, big[pick], precision)) == (narrow, 256)


@pytest.mark.parametrize("deck,size,precision,n,widths", [
    (mesh, 200, lanes.PREC_MIXED, 700, (256, 128)), (mesh, 200, lanes.PREC_FP64, 1500, (256, 128)),
    (mesh, 1000, lanes.PREC_FP64, 300, (512, 256)), (mesh, 1000, lanes.PREC_MIXED, 1000, (512, 256))])
def test_calls_after_another_width(deck, size, precision, n, widths):
    """A batch on a context that solved one lane at another width runs there at
    first and changes over later: the same bits in every call."""
    fr, slots, values = deck(size)
    v = values(n)
    assert (width(fr, slots, v[:1], precision), width(fr, slots, v, precision)) == widths
    want = solve(fr, slots, v, precision, lanes.PATH_BLOCK)
    ctx = lanes.DcLanes(fr)
    ctx.set_mode(precision=precision, path=lanes.PATH_BLOCK)
    ctx.set_lanes(slots, v[:1])
    ctx.solve(x0=np.zeros(fr.n))
    ctx.set_lanes(slots, v)
    for _ in range(8):
        x, it, st, _ = ctx.solve(x0=np.zeros(fr.n))
        for u, w in zip((x.view(np.uint64), it, st), want):
            assert np.array_equal(u, w)
    ctx.close()


@pytest.mark.parametrize("precision", [lanes.PREC_FP64, lanes.PREC_MIXED])
def test_broad_transients_equal_wide(precision):
    """A digital block's transient lanes with an SM each (512 threads) and one
    lane more (256)."""
    fr, slots = decks.digital_block(size=1500, n_cells=37, n_inputs=8)
    v = decks.digital_block_vto(len(slots), 149, seed=3)
    out = []
    for n in (149, 148):
        ctx = lanes.DcLanes(fr)
        ctx.set_mode(precision=precision, path=lanes.PATH_BLOCK)
        ctx.set_lanes(slots, v[:n])
        stats, x = ctx.tran(lanes.tran_opts(2e-11, 1e-11, 1e-11))[3:5]
        out.append((x.view(np.uint64)[:148], stats[:148]))
        assert ctx.block_info()["width"] == (256 if n == 149 else 512)
        ctx.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("deck,size", [(ladder, 1), (ladder, 28), (ladder, 29), (ladder, 61), (grid, 0), (mesh, 50),
                                       (mesh, 110), (mesh, 140)])
def test_block_lanes_equal_warp_lanes(deck, size):
    fr, slots, values = deck(size)
    v = values(17)
    a = solve(fr, slots, v, lanes.PREC_FP64, lanes.PATH_WARP)
    b = solve(fr, slots, v, lanes.PREC_FP64, lanes.PATH_BLOCK)
    for u, w in zip(a, b):
        assert np.array_equal(u, w)


def crowd(nodes, parts):
    """A few nodes with thousands of resistors between them: a small tape
    beside lanes that take all of a CTA's shared memory."""
    c = Circuit()
    c.V("vin", "n0", "0", dc=1.0)
    for k in range(parts):
        i = k % nodes
        j = (i + 1 + k // nodes % (nodes - 1)) % nodes
        c.R(f"r{k}", f"n{i}", f"n{j}" if k % 3 else "0", 100.0 + k % 71)
    c.D("d0", f"n{nodes - 1}", "0", is_=1e-14, n=1.0, rs=10.0)
    fr = c.freeze()
    return fr, [fr.slot("vin", "dc")]


# (the two smallest, whose rows of single ops take less than a ring, one part at
# a time: the last few read their words where they lie)
@pytest.mark.parametrize("nodes,first,last,step", [(9, 2460, 2960, 90), (20, 2070, 2400, 90), (2, 1452, 1468, 1),
                                                   (3, 1690, 1702, 1)])
def test_lanes_that_fill_shared_memory(nodes, first, last, step):
    """Every count of parts up to `last` is a warp lane, whether its words lie
    in shared memory, stream through a ring or are read where they lie; DC
    solves, alone and in a group, equal the block lanes', sweeps and measured
    transients run or are refused."""
    import torch
    tran = lanes.tran_opts(1e-9, 1e-10, 1e-10)
    v = np.linspace(0.5, 3.0, 3).reshape(-1, 1)
    for parts in list(range(first, last, step)) + [last]:
        fr, slots = crowd(nodes, parts)
        a = solve(fr, slots, v, lanes.PREC_FP64, lanes.PATH_WARP)
        b = solve(fr, slots, v, lanes.PREC_FP64, lanes.PATH_BLOCK)
        for u, w in zip(a, b):
            assert np.array_equal(u, w), parts
        ctx = lanes.DcLanes(fr)
        ctx.set_mode(precision=lanes.PREC_FP64, path=lanes.PATH_WARP)
        ctx.set_lanes(slots, v)
        pts = np.linspace(0.0, 1.0, 3)
        try:
            x, it, cv, st, _ = ctx.sweep(slots[0], pts)
        except lanes.LaneError as e:  # (a sweep's lane is a little larger)
            assert e.code == lanes.ESL_NOT_ELIGIBLE and parts > last - 5, str(e)
        else:
            xo, ito, cvo = oracle.dc_sweep(fr, slots[0], pts)
            assert (st == lanes.SWEEP_DONE).all() and np.array_equal(it[0], ito) and cv.all() and all(cvo)
            assert np.allclose(x[0], xo, rtol=1e-9, atol=1e-12)
        for n_meas in (1, 30):
            try:
                ctx.tran_meas(tran, [lanes.window(lanes.MEAS_MAX, fr.unknown("n1"))] * n_meas)
            except lanes.LaneError as e:
                assert e.code == lanes.ESL_NOT_ELIGIBLE, str(e)
        x = torch.zeros((2, 3, fr.n), dtype=torch.float64, device="cuda")
        words = torch.zeros((2, 2, 3), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        other = lanes.DcLanes(fr)
        other.set_mode(precision=lanes.PREC_FP64, path=lanes.PATH_WARP)
        other.set_lanes(slots, v)
        lanes.group_solve_device([ctx, other], [x[k].data_ptr() for k in range(2)],
                                 [words[0, k].data_ptr() for k in range(2)],
                                 [words[1, k].data_ptr() for k in range(2)], cold=[False] * 2)
        ctx.close()
        other.close()
        for k in range(2):
            assert np.array_equal(x[k].cpu().numpy().view(np.uint64), a[0]), parts


def test_wide_words_equal_the_oracle():
    """A mesh of 2,500 unknowns: past 65,536 values."""
    fr, slots, values = mesh(2500)
    v = values(2)
    ctx = lanes.DcLanes(fr)
    ctx.set_mode(precision=lanes.PREC_FP64, path=lanes.PATH_BLOCK)
    ctx.set_lanes(slots, v)
    x, it, st, _ = ctx.solve(x0=np.zeros(fr.n))
    assert ctx.block_info()["ntv"] + fr.n + 3 >= 65536
    ctx.close()
    xo, ito, cv = oracle.dc_points(fr, slots, v, warm=np.zeros(fr.n))
    assert np.array_equal(st == lanes.LANE_CONVERGED, cv.astype(bool)) and np.array_equal(it, ito)
    assert np.array_equal(x.view(np.uint64), xo.view(np.uint64))


@pytest.mark.parametrize("epochs", [1, 2, 3, 5])
def test_graph_steps_equal_single_steps(epochs):
    """Equal rows (any order the same batch): a run of several steps, all but
    the first replayed, ends in the weights of as many runs of one."""
    import torch
    x = torch.full((16, 5), 0.3, device="cuda") * torch.arange(1, 6, device="cuda")
    y = torch.full((16, 19), 0.7, device="cuda") - 0.1 * torch.arange(19, device="cuda")
    torch.cuda.synchronize()
    one, many = (mlp.Mlp(5, 32, 3, 19, seed=4) for _ in range(2))
    la = many.train(x.data_ptr(), y.data_ptr(), 16, epochs=epochs, batch=16, lr=1e-2)
    lb = [one.train(x.data_ptr(), y.data_ptr(), 16, epochs=1, batch=16, lr=1e-2)[0] for _ in range(epochs)]
    assert np.array_equal(la, np.array(lb, np.float32))
    for (wa, ba), (wb, bb) in zip(many.weights(), one.weights()):
        assert np.array_equal(wa, wb) and np.array_equal(ba, bb)
    one.close()
    many.close()


@pytest.mark.parametrize("deck", ["ring", "grid"])
def test_compiled_lu_without_the_factors(deck):
    """dx and the verdicts with and without the factors' planes, a dead pivot
    and a tiny matrix among the lanes."""
    import torch
    fr = decks.ring_oscillator(lanes=2)[0] if deck == "ring" else decks.grid_diodes(seed=1)[0]
    cp, ri = lanes.pattern(fr)
    rng = np.random.default_rng(3)
    lead = rng.uniform(0.5, 2.0, len(ri)) * rng.choice((-1.0, 1.0), len(ri))
    diag = np.array([np.searchsorted(ri[cp[j]:cp[j + 1]], j) + cp[j] for j in range(fr.n)])
    lead[diag] += 8.0
    n = 131
    vals = lead[:, None] * rng.uniform(0.8, 1.2, (len(ri), n))
    vals[diag[3], 5] = 0.0
    vals[:, 7] *= 1e-9
    vals[diag[2], 9] = np.inf
    a = torch.tensor(vals, device="cuda")
    rhs = torch.tensor(rng.normal(size=(fr.n, n)), device="cuda")
    dx = [torch.zeros((fr.n, n), dtype=torch.float64, device="cuda") for _ in range(2)]
    bad = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2)]
    ctx = lanes.DcLanes(fr)
    torch.cuda.synchronize()
    ctx.lu_lanes_compiled(lead, a.data_ptr(), rhs.data_ptr(), dx[0].data_ptr(), bad[0].data_ptr(), n)
    tv = torch.zeros((ctx.tape_size()[2], n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.lu_lanes_compiled(lead, a.data_ptr(), rhs.data_ptr(), dx[1].data_ptr(), bad[1].data_ptr(), n, tv.data_ptr())
    ctx.close()
    b = [v.cpu().numpy() for v in bad]
    assert np.array_equal(b[0], b[1]) and b[0].any() and not b[0].all()
    x = [v.cpu().numpy()[:, b[0] == 0].view(np.uint64) for v in dx]
    assert np.array_equal(x[0], x[1])
