"""Uneven batching and the lanes-per-CTA autotuner (B200).

Three circuits of different sizes and lane counts solved in one launch give
each lane bitwise the result of its own context's launch (the same per-lane
solve on the same tape); the autotuner's choice of lanes per CTA changes
timing only, never a result bit.
"""

import numpy as np
import pytest

from espice_b200 import decks, lanes

pytestmark = pytest.mark.gpu


def _case(rows, cols, n_diodes, points, seed):
    fr, slots, values = decks.grid_diodes(seed=seed, rows=rows, cols=cols, n_diodes=n_diodes, points=points)
    ctx = lanes.DcLanes(fr)
    ctx.set_lanes(slots, values)
    return fr, ctx


def test_group_launch_matches_single_launches():
    import torch
    cases = [_case(4, 4, 3, 37, 1), _case(8, 8, 16, 256, 2), _case(10, 12, 20, 100, 3)]
    opts = lanes.newton_opts()
    singles = []
    for fr, ctx in cases:
        x, it, st, _ = ctx.solve(x0=np.zeros(fr.n), opts=opts)
        singles.append((x, it, st))
    bufs = []
    for fr, ctx in cases:
        bufs.append((torch.zeros((ctx.n_lanes, fr.n), dtype=torch.float64, device="cuda"),
                     torch.zeros(ctx.n_lanes, dtype=torch.int32, device="cuda"),
                     torch.zeros(ctx.n_lanes, dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    stats = lanes.group_solve_device([c for _, c in cases], [b[0].data_ptr() for b in bufs],
                                     [b[1].data_ptr() for b in bufs], [b[2].data_ptr() for b in bufs], opts=opts)
    torch.cuda.synchronize()
    for (x, it, st), (dx, di, ds), s, (fr, ctx) in zip(singles, bufs, stats, cases):
        assert np.array_equal(dx.cpu().numpy().view(np.uint64), x.view(np.uint64))
        assert np.array_equal(di.cpu().numpy().astype(np.uint32), it)
        assert np.array_equal(ds.cpu().numpy().astype(np.uint32), st)
        assert s["lanes"] == ctx.n_lanes and s["converged"] == int((st == lanes.LANE_CONVERGED).sum())
    for _, ctx in cases:
        ctx.close()


def test_autotune_keeps_results():
    fr, ctx = _case(8, 8, 16, 512, 4)
    x0 = np.zeros(fr.n)
    x1, it1, st1, _ = ctx.solve(x0=x0)
    best = ctx.autotune(x0=x0)
    assert best in (1, 2, 4, 8)
    x2, it2, st2, _ = ctx.solve(x0=x0)
    assert np.array_equal(x1.view(np.uint64), x2.view(np.uint64))
    assert np.array_equal(it1, it2) and np.array_equal(st1, st2)
    ctx.close()


@pytest.mark.parametrize("precision", [lanes.PREC_FP64, lanes.PREC_MIXED])
def test_block_group_uneven_batch_against_oracle(precision):
    """The uneven batch on the block lanes: the eight mesh-with-gates
    topologies (50 to 2,000 unknowns), six supply values each, in one launch
    (work items largest topology first; the largest are most of the work and
    lie in global memory, so all do). FP64: every lane bitwise the oracle, the same
    iteration counts. Mixed: the oracle's convergence, values within 1e-9
    relative or 1e-12 absolute."""
    import torch
    import parity
    from oracle import oracle
    vals = np.linspace(0.8, 1.8, 6).reshape(-1, 1)
    ctxs, bufs, decks_ = [], [], []
    for size in decks.MESH_GATES_SIZES:
        fr, slots = decks.mesh_gates(size)
        c = lanes.DcLanes(fr)
        c.set_mode(precision=precision, path=lanes.PATH_BLOCK)
        c.set_lanes(slots, vals)
        ctxs.append(c)
        decks_.append((fr, slots))
        bufs.append((torch.zeros((len(vals), fr.n), dtype=torch.float64, device="cuda"),
                     torch.zeros(len(vals), dtype=torch.int32, device="cuda"),
                     torch.zeros(len(vals), dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    stats = lanes.group_solve_device(ctxs, [b[0].data_ptr() for b in bufs], [b[1].data_ptr() for b in bufs],
                                     [b[2].data_ptr() for b in bufs], cold=[True] * len(ctxs))
    torch.cuda.synchronize()
    for (fr, slots), b, s, c in zip(decks_, bufs, stats, ctxs):
        assert s["path"] == lanes.PATH_BLOCK
        x = b[0].cpu().numpy()
        it = b[1].cpu().numpy().astype(np.uint32)
        st = b[2].cpu().numpy().astype(np.uint32)
        xo, ito, cvo = oracle.dc_points(fr, slots, vals, warm=None)
        conv = st == lanes.LANE_CONVERGED
        if precision == lanes.PREC_FP64:
            assert parity.assert_dc_parity(fr, slots, vals, None, oracle.newton_opts(), x, it, conv, xo, ito, cvo,
                                           f"group n={fr.n}") == 1.0
        else:
            assert np.array_equal(conv, cvo.astype(bool))
            assert parity.close(x[conv], xo[conv]).all(), float(np.max(np.abs(x[conv] - xo[conv])))
        c.close()


@pytest.mark.parametrize("precision", [lanes.PREC_FP64, lanes.PREC_MIXED])
@pytest.mark.parametrize("sizes,counts", [
    ((50, 100, 200), (40, 40, 40)),      # all in shared memory
    ((50, 200, 1500), (300, 300, 4)),    # the small ones there, the large one in global memory
    ((200, 2500), (400, 2)),             # and its words of the wide form, for one ring
    ((50, 200, 1500), (4, 4, 8)),        # all in global memory
])
def test_block_group_placements(sizes, counts, precision):
    """Where a group's working sets lie changes no bit: its lanes are those of
    each topology solved alone."""
    import torch
    ctxs, bufs, alone = [], [], []
    for size, n in zip(sizes, counts):
        fr, slots = decks.mesh_gates(size)
        c = lanes.DcLanes(fr)
        c.set_mode(precision=precision, path=lanes.PATH_BLOCK)
        c.set_lanes(slots, np.linspace(0.8, 1.8, n).reshape(-1, 1))
        alone.append(c.solve(x0=None)[:3])
        ctxs.append(c)
        bufs.append((torch.zeros((n, fr.n), dtype=torch.float64, device="cuda"),
                     torch.zeros(n, dtype=torch.int32, device="cuda"),
                     torch.zeros(n, dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    lanes.group_solve_device(ctxs, [b[0].data_ptr() for b in bufs], [b[1].data_ptr() for b in bufs],
                             [b[2].data_ptr() for b in bufs], cold=[True] * len(ctxs))
    for c, b, (x, it, st) in zip(ctxs, bufs, alone):
        assert np.array_equal(b[0].cpu().numpy().view(np.uint64), x.view(np.uint64))
        assert np.array_equal(b[1].cpu().numpy(), it) and np.array_equal(b[2].cpu().numpy(), st)
        c.close()
