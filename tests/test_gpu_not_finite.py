"""Positions that the mixed form's 32-bit coordinates cannot hold.

A coordinate wraps at a window of the box and ten bits of the window's index tell motion
by whole windows; a position that is not a number, infinite or a multiple of 1,024 windows
away looks like one that has not moved.  A position that is not a number must end the run
with E_NAN, as the NaN forces it causes do in the reference (src/md_simulator.cpp:646-652);
a far one must rebuild the list (src/neighborlist.cpp:134-143).
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def fluid(cells):
    rng = np.random.default_rng(5)
    pos, box = W.fcc_lattice(cells, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    return pos, np.zeros_like(pos), np.zeros(len(pos), np.int32), W.lj_params(box)


# 5 cells: the step kernel; 24 cells: graphs of single kernels, or kernels launched one by one
@pytest.mark.parametrize("cells,spg", [((5, 5, 5), 0), ((5, 5, 5), -1), ((24, 24, 24), 0), ((24, 24, 24), -1)])
@pytest.mark.parametrize("integrator", [0, 1, 2])
def test_position_that_is_not_a_number_ends_the_run(cells, spg, integrator):
    pos, vel, typ, p = fluid(cells)
    p = dict(p, integrator=integrator, lang_friction=1.0, seed=1)
    vel[3, 1] = np.nan
    s = G.System(pos, vel, typ, p, precision=G.MIXED, steps_per_graph=spg)
    s.setup()
    with pytest.raises(G.CavError) as e:
        s.step(20)
    assert e.value.status == G.E_NAN
    assert s.stats()["steps"] <= 2  # at the force of the step that met it, seen by the next step at the latest
    s.close()


# windows of a box of 5 and of 30 cells: the whole box, four of 12.6
@pytest.mark.parametrize("cells", [(5, 5, 5), (30, 5, 5)])
@pytest.mark.parametrize("windows", [1024.0, -2048.0, 1024.0 * 2 ** 20, 1024.0 * 2 ** 40, np.inf])
def test_far_displacement_rebuilds(cells, windows):
    pos, vel, typ, p = fluid(cells)
    ce = p["nl_cutoff"] * p["nl_coef"]
    L = p["hi"][0] - p["lo"][0]
    width = L / max(np.floor(L / (4 * ce)), 1.0)
    i = int(np.argmin(np.abs(pos[:, 0])))  # the atom nearest the lower face: coordinate and window 0
    vel[i, 0] = windows * width / p["dt"]
    pos[i, 0] = 0.0
    s = G.System(pos, vel, typ, p, precision=G.MIXED)
    s.setup()
    s.step(1)
    assert s.stats()["rebuilds"] == 2  # set-up and the step's own
    assert np.abs(s.state()[2][i]).max() == 0.0  # out of the others' reach
    s.close()


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("cells,spg", [(3, 0), (3, -1), (12, 0)])
def test_position_that_is_not_a_number_of_an_atom_on_its_own(cells, spg, precision):
    """Without neighbours it causes no NaN force, and its displacement is not "more than" half the
    skin: the others go on, the list stays."""
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos, vel = (g + 0.5) * 4.0, np.zeros((cells ** 3, 3))
    vel[2, 0] = np.nan
    s = G.System(pos, vel, np.zeros(len(pos), np.int32), W.lj_params(np.full(3, 4.0 * cells)), precision=precision,
                 steps_per_graph=spg)
    s.setup()
    s.step(10)
    x, _, a = s.state()
    assert s.stats()["rebuilds"] == 1 and s.stats()["steps"] == 10
    assert np.isnan(x[2, 0]) and np.isfinite(np.delete(x, 2, 0)).all() and (a == 0.0).all()
    s.close()
