"""The mixed form's fixed-point coordinates at the edges of their range.

The pair kernel takes displacements from 32-bit integers that wrap at a window of the
box (the whole box when it is short, several windows of at least four list cutoffs when
it is long).  Checked against the FP64 form from the same start: the smallest box a
context accepts, long boxes of several windows, boxes far from the origin; and a
displacement of a whole window in one step, which the integers alone do not show but
which must rebuild the list.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fluid(cells, shift=0.0, seed=5):
    import workloads as W

    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice(cells, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.12, 0.12, size=pos.shape), box)
    pos[pos >= box] = 0.0
    params = W.lj_params(box)
    params["lo"], params["hi"] = np.full(3, shift), box + shift
    return pos + shift, W.thermal_velocities(len(pos), 1.44, rng), np.zeros(len(pos), np.int32), params


# 4 cells: edges of 6.72, just above two list cutoffs (5.6); 30 cells: 50.4, four windows of
# 12.6; the shifts leave FP64 positions with an ulp of 2^-43 and 2^-33
@pytest.mark.parametrize("cells,shift", [((4, 4, 4), 0.0), ((30, 4, 5), 0.0), ((5, 7, 14), -1000.0),
                                         ((4, 30, 13), 1.0e6)])
def test_forces_and_steps_follow_the_fp64_form(cells, shift):
    import cavgpu as G

    pos, vel, typ, params = fluid(cells, shift)
    got = []
    for precision in (G.MIXED, G.FP64):
        s = G.System(pos, vel, typ, params, precision=precision)
        s.setup()
        a0 = s.state()[2]
        s.step(40)
        got.append((a0,) + s.state())
        s.close()
    (a, x, v, _), (ar, xr, vr, _) = got
    assert np.sqrt(((a - ar) ** 2).sum() / (ar ** 2).sum()) < 1e-5  # the mixed form's force bar
    # that bar on |a| ~ 100 (rms) over t = 0.2 is 2e-5 in position, times the growth of a
    # perturbation in a dense fluid over that time (under 5); an ulp of the shifted positions adds less
    L = params["hi"] - params["lo"]
    dx = x - xr - np.round((x - xr) / L) * L
    assert np.abs(dx).max() < 1e-4 and np.abs(v - vr).max() < 1e-3


@pytest.mark.parametrize("windows", [1, 2, -1])
def test_displacement_of_whole_windows_rebuilds(windows):
    import cavgpu as G

    pos, vel, typ, params = fluid((30, 5, 5))
    ce = params["nl_cutoff"] * params["nl_coef"]
    L = params["hi"][0] - params["lo"][0]
    width = L / np.floor(L / (4 * ce))
    vel[:] = 0.0  # one atom crosses whole windows in one step, the others hardly move
    i = int(np.argmin(np.abs(pos[:, 0] - 0.5 * L)))
    vel[i, 0] = windows * width / params["dt"]
    acc = []
    for precision in (G.MIXED, G.FP64):
        s = G.System(pos, vel, typ, params, precision=precision)
        s.setup()
        s.step(1)
        assert s.stats()["rebuilds"] == 2  # set-up and the step's own
        acc.append(s.state()[2])
        s.close()
    # the atom lands on top of others: compare the atoms it does not touch (|a| within reason)
    calm = np.abs(acc[1]).max(1) < 1e4
    assert calm.sum() > 0.9 * len(pos)
    assert np.sqrt(((acc[0] - acc[1])[calm] ** 2).sum() / (acc[1][calm] ** 2).sum()) < 1e-5
