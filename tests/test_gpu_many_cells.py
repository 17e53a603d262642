"""Boxes of more than 2^27 search cells, most of them empty.

The kernel that sorts cells and moves the atoms' state runs a warp per cell: thread numbers
beyond 32 bits.  A droplet that sits across the corner of a 1440-wide box (514 cells per axis)
has atoms in the last cells as well as in the first; it must move as the same droplet in a box
of 40.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
def test_droplet_across_the_corner_of_a_large_box(precision):
    rng = np.random.default_rng(2)
    pos, box = W.fcc_lattice((6, 6, 6), 0.8442)
    pos = pos - box / 2 + rng.uniform(-0.1, 0.1, size=pos.shape)
    vel = W.thermal_velocities(len(pos), 1.0, rng)
    out = []
    for edge in (40.0, 1440.0):
        L = np.full(3, edge)
        x = np.mod(pos, L)
        x[x >= L] = 0.0
        s = G.System(x, vel, np.zeros(len(pos), np.int32), W.lj_params(L), precision=precision)
        s.setup()
        a0 = s.state()[2]
        s.step(25)
        p, v, _ = s.state()
        out.append((a0, p - np.round(p / L) * L, v, s.stats()["rebuilds"]))
        s.close()
    (a, p, v, r), (A, P, V, R) = out
    assert r == R > 1
    # positions by the far faces are rounded to 2^-42: times the force's slope (1e3) 2e-10 in
    # FP64; the mixed form's unit is 3e-9, and its forces are good to 1e-5 of the rms
    tol = 1e-8 if precision == G.FP64 else 1e-4 * np.sqrt((a ** 2).mean())
    assert np.abs(a - A).max() < tol
    assert np.abs(p - P).max() < 1e-3 * tol + 1e-9 and np.abs(v - V).max() < 0.1 * tol + 1e-8


def test_more_cells_than_the_stated_maximum_are_refused():
    pos = np.random.default_rng(0).random((8, 3)) * 100
    for edge in (2900.0, 4600.0):  # 1035^3 > 2^30; 1642^3 > 2^32
        L = np.full(3, edge)
        with pytest.raises(G.CavError) as e:
            G.System(pos, np.zeros((8, 3)), np.zeros(8, np.int32), W.lj_params(L))
        assert e.value.status == G.E_RANGE
