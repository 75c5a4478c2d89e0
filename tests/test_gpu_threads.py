"""Contexts on several host threads at once, of circuits whose kernels take
different amounts of shared memory (B200): no call fails, and every thread
gets its lanes' bits each time. (A kernel's shared-memory limit is the
process's: set per launch, two of a hundred calls here failed.)"""

import threading

import numpy as np
import pytest

from espice_b200 import decks, lanes

pytestmark = pytest.mark.gpu


def test_threads_with_contexts_of_their_own():
    jobs = [(50, 30, lanes.PATH_BLOCK), (200, 500, lanes.PATH_BLOCK), (400, 40, lanes.PATH_BLOCK),
            (400, 700, lanes.PATH_BLOCK), (50, 700, lanes.PATH_BLOCK), (200, 40, lanes.PATH_BLOCK),
            (30, 64, lanes.PATH_WARP), (100, 64, lanes.PATH_WARP)]
    errors = []

    def work(size, n, path):
        try:
            fr, slots = decks.mesh_gates(size)
            ctx = lanes.DcLanes(fr)
            ctx.set_mode(precision=lanes.PREC_FP64, path=path)
            ctx.set_lanes(slots, np.linspace(0.8, 1.8, n).reshape(-1, 1))
            first = None
            for _ in range(200):
                x = ctx.solve(x0=np.zeros(fr.n))[0].view(np.uint64)
                first = x if first is None else first
                assert np.array_equal(first, x)
            ctx.close()
        except Exception as e:
            errors.append((size, n, str(e)))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
