"""Pair forces act between an atom and the image its list names.

A force cutoff beyond the neighbour cutoff is legal (the reference's own two-atom demo
has a list cutoff of 5 and a force cutoff of 10, tests/t001_lj.cpp).  In a box hardly wider than
two list cutoffs a listed pair may drift further apart than half the box before the list
is rebuilt; the mixed form must go on with the listed image, as the reference and the FP64
form do, and not with the one that is now nearer.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def gas(edges, n, seed):
    """Atoms at least 0.95 apart."""
    rng, L = np.random.default_rng(seed), np.array(edges)
    pos = np.empty((0, 3))
    while len(pos) < n:
        p = rng.random(3) * L
        d = pos - p
        d -= np.round(d / L) * L
        if not len(pos) or (d ** 2).sum(1).min() > 0.9:
            pos = np.vstack([pos, p])
    return pos, L


# list cutoff 2.8, skin 0.3: edges of 5.62 to 6.2 let listed pairs drift past half the box;
# 23 long: two windows on that axis, one on the others
@pytest.mark.parametrize("edges,n", [((5.62, 5.62, 5.62), 60), ((5.7, 6.1, 30.0), 300), ((23.0, 5.65, 8.0), 300)])
@pytest.mark.parametrize("types", [1, 2])
@pytest.mark.parametrize("kw", [{}, {"steps_per_graph": -1}, {"tpa": 1}, {"force_kernel": 2}],
                         ids=["default", "single", "one-lane", "segments"])
def test_mixed_follows_the_listed_image(edges, n, types, kw):
    pos, L = gas(edges, n, 7)
    more = {}
    if types == 2:
        more = dict(ntypes=2, eps=np.array([[1.0, 0.7], [0.7, 0.5]]), sigma=np.array([[1.0, 0.9], [0.9, 0.85]]))
    p = W.lj_params(L, dt=0.002, **more)
    p["lj_cutoff"] = 4.5
    typ = (np.arange(n) % types).astype(np.int32)
    vel = W.thermal_velocities(n, 1.0, np.random.default_rng(1))
    m = G.System(pos, vel, typ, p, precision=G.MIXED, **kw)
    r = G.System(pos, vel, typ, p, precision=G.FP64)
    worst = 0.0
    for s in (m, r):
        s.setup()
    np.testing.assert_array_equal(m.pairs(), r.pairs())
    for _ in range(12):
        for s in (m, r):
            s.step(4)
        a, b = m.state()[2], r.state()[2]
        worst = max(worst, np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))
    assert m.stats()["rebuilds"] == r.stats()["rebuilds"] > 1
    m.close(), r.close()
    # a pair taken at the wrong image changes its force by the whole pair force, ~1e-2 of the
    # rms and more; FP32 forces part from FP64 by 1e-6, 48 steps of a dilute gas add tenfold
    assert worst < 1e-4


def test_batch_of_narrow_and_wide_boxes():
    systems = []
    for k, (edges, n) in enumerate([((5.62, 5.62, 5.62), 60), ((23.0, 12.0, 8.0), 500), ((5.65, 26.0, 6.0), 250)]):
        pos, L = gas(edges, n, 20 + k)
        vel = W.thermal_velocities(n, 1.0, np.random.default_rng(k))
        systems.append((pos, vel, np.zeros(n, np.int32), np.zeros(3), L))
    p = W.lj_params(systems[0][4], dt=0.002)
    p["lj_cutoff"] = 4.5
    acc = []
    for precision in (G.MIXED, G.FP64):
        s = G.Batch(systems, p, precision=precision)
        s.setup()
        out = []
        for _ in range(12):
            s.step(4)
            out.append(s.split(s.state()[2]))
        acc.append(out)
        s.close()
    for a, b in zip(*acc):
        for x, y in zip(a, b):
            assert np.sqrt(((x - y) ** 2).sum() / (y ** 2).sum()) < 1e-4
