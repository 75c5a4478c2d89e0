"""The block lanes' task streams on the CPU: task_streams.cpp packs a tape
and runs the streams as the kernels do, every warp from barrier to barrier.
Each op once and in its value's order (the values are the sequential replay's
bit for bit), the same barriers for every warp, no value that two warps touch
between two of them; for tapes of few unknowns and of thousands, compact and
wide words, both orders of the ready tasks, diagonally dominant and with
pivoting leads. And where the rows are bound by their number, a row's tasks
are neighbours: their loads fall into few sectors."""

import os
import subprocess

import numpy as np
import pytest

from espice_b200 import decks, lanes
from espice_b200.circuit import Circuit

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "espice_b200", "csrc")


@pytest.fixture(scope="module")
def streams(tmp_path_factory):
    d = tmp_path_factory.mktemp("streams")
    exe = str(d / "task_streams")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", SRC, "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "task_streams.cpp"), os.path.join(SRC, "host", "schedule.cpp"),
                    os.path.join(SRC, "host", "sparse.cpp"), "-o", exe], check=True)

    def go(fr, seed=1, dominant=True):
        cp, ri = lanes.pattern(fr)
        rng = np.random.default_rng(seed)
        lead = rng.uniform(0.5, 2.0, len(ri)) * rng.choice((-1.0, 1.0), len(ri))
        diag = [cp[j] + np.searchsorted(ri[cp[j]:cp[j + 1]], j) for j in range(fr.n)]
        if dominant:
            lead[diag] += 8.0
        vals = lead * rng.uniform(0.9, 1.1, len(ri))
        rhs = rng.normal(size=fr.n) * (rng.random(fr.n) < 0.7)  # some zero: the solves skip them
        path = str(d / "tape.bin")
        with open(path, "wb") as f:
            np.array([fr.n], np.uint32).tofile(f)
            cp.astype(np.uint32).tofile(f)
            ri.astype(np.uint32).tofile(f)
            for a in (lead, vals, rhs):
                a.astype(np.float64).tofile(f)
        out = subprocess.run([exe, path], check=True, capture_output=True, text=True).stdout.split("\n")
        rows = [line.split() for line in out if line]
        assert len(rows) == 3 and all(r[0] == "ok" for r in rows), out
        return {int(r[1]): (int(r[2]), float(r[3])) for r in rows}
    return go


def lone():
    c = Circuit()
    c.I("i0", "0", "n0", dc=1e-3)
    c.R("r0", "n0", "0", 1e3)
    return c.freeze()


@pytest.mark.parametrize("deck", [lone, lambda: decks.ring_oscillator(lanes=1)[0], lambda: decks.grid_diodes(seed=1)[0],
                                  lambda: decks.mesh_gates(50)[0], lambda: decks.mesh_gates(400)[0],
                                  lambda: decks.analog_block()[0], lambda: decks.mesh_gates(1000)[0],
                                  lambda: decks.mesh_gates(2500)[0]],
                         ids=["one", "ring", "grid", "mesh50", "mesh400", "analog", "mesh1000", "mesh2500"])
@pytest.mark.parametrize("dominant", [True, False])
def test_streams_run_the_replay(streams, deck, dominant):
    try:
        streams(deck(), dominant=dominant)
    except subprocess.CalledProcessError:
        assert not dominant  # a random lead may be singular


@pytest.mark.parametrize("deck", [lambda: decks.digital_block(size=2000, n_cells=50, n_inputs=8)[0],
                                  lambda: decks.mesh_gates(2000)[0]], ids=["digital2000", "mesh2000"])
def test_neighbours_where_rows_are_many(streams, deck):
    """About one sector an update, of up to 7/3 (FP64)."""
    for warps, (rows, sectors) in streams(deck()).items():
        assert sectors < 1.25, (warps, rows, sectors)
