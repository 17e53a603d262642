"""Small contexts stepped at the same time from several threads.

The step kernel's grid then leaves room for the other contexts; every context must move, and
record, as it does alone.
"""
import threading

import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def context(cells, precision, integrator, seed):
    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    p = W.lj_params(box, integrator=integrator, friction=1.0, seed=seed)
    s = G.System(pos, W.thermal_velocities(len(pos), 1.0, rng), np.zeros(len(pos), np.int32), p, precision=precision)
    s.setup()
    return s


# sizes whose grids differ alone, beside one other context and beside many
@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("threads", [2, 6])
def test_threads_step_their_contexts_as_alone(precision, threads):
    shapes = [(5, 0), (10, 1), (13, 0), (7, 2), (12, 1), (14, 0)][:threads]
    out = []
    for together in (False, True):
        ctx = [context(c, precision, i, 3 + k) for k, (c, i) in enumerate(shapes)]
        rec = [None] * threads

        def work(k):
            rec[k] = ctx[k].run(300, 10)

        if together:
            th = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
            for t in th:
                t.start()
            for t in th:
                t.join()
        else:
            for k in range(threads):
                work(k)
        out.append([(r, *s.state(), s.stats()["rebuilds"]) for r, s in zip(rec, ctx)])
        for s in ctx:
            s.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
