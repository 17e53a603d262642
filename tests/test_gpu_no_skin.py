"""Lists without a skin (cutoff_extra_coef = 1): any motion rebuilds, rest does not.

The half-skin test is "displacement^2 > 0" then (src/neighborlist.cpp:134-143, 318).
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("cells,spg", [(5, 0), (5, -1), (24, 0)])
@pytest.mark.parametrize("coef", [1.0, 1.0 + 1e-9])
def test_rebuilds_without_a_skin(moving, cells, spg, coef):
    # atoms at rest, far from one another
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    L = np.full(3, 3.0 * cells)
    pos = (g + 0.5) * 3.0
    vel = np.zeros_like(pos)
    if moving:
        vel[1, 0] = 1e-3
    p = W.lj_params(L, dt=0.002)
    p["nl_coef"] = coef
    got = []
    for precision in (G.MIXED, G.FP64):
        s = G.System(pos, vel, np.zeros(len(pos), np.int32), p, precision=precision, steps_per_graph=spg)
        s.setup()
        s.step(20)
        got.append(s.stats()["rebuilds"])
        s.close()
    assert got[0] == got[1] == (21 if moving else 1)
