"""Small systems in boxes with many more cells than atoms.

The step kernel scans a replica's cells in one block, so boxes of many cells must run as
graphs of kernels however few their atoms; a droplet on either side of that line moves as
with kernels launched one by one.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


# 21^3 = 9,261 cells; 23^3 = 12,167 and 24^3 = 13,824, either side of the line; 35^3 = 42,875
@pytest.mark.parametrize("edge,cells", [(60.0, 21), (65.0, 23), (68.0, 24), (100.0, 35)])
@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
def test_droplet_in_a_sparse_box(edge, cells, precision):
    rng = np.random.default_rng(2)
    pos, box = W.fcc_lattice((6, 6, 6), 0.8442)
    L = np.full(3, edge)
    assert int(edge / 2.8) == cells
    pos = np.mod(pos - box / 2 + rng.uniform(-0.1, 0.1, size=pos.shape), L)
    pos[pos >= edge] = 0.0
    vel = W.thermal_velocities(len(pos), 1.0, rng)
    out = []
    for spg in (0, -1):
        s = G.System(pos, vel, np.zeros(len(pos), np.int32), W.lj_params(L), precision=precision, steps_per_graph=spg)
        s.setup()
        rec = s.run(40, 4)
        out.append((s.state(), rec, s.stats()))
        s.close()
    assert (out[0][2]["graph_launches"] > 0) == (cells ** 3 > 12288)
    assert out[0][2]["rebuilds"] == out[1][2]["rebuilds"] > 1
    np.testing.assert_array_equal(out[0][1], out[1][1])
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
