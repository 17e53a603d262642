"""The FP64 form's pair exchange (every pair evaluated once) against the full-list kernel.

Eight lanes per atom run the full-list kernel, which evaluates a pair from both sides; one,
two and four lanes run the exchange and must agree with one another bit for bit, and with
the full list to rounding.  Sizes at the edges of its parts: fewer atoms than a warp, a
task more or less than a whole number, the smallest box (every pair crosses a face
somewhere), two types with their own cutoffs, rows long enough to outgrow the space of the
claimed entries.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fluid(cells, vacant, rho=0.8442, types=1, integrator=0, seed=11):
    import workloads as W

    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice(cells, rho)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape) * (0.8442 / rho) ** (1 / 3), box)
    pos[pos >= box] = 0.0
    keep = np.sort(rng.permutation(len(pos))[vacant:])
    pos = pos[keep]
    kw = {}
    if types == 2:
        sig = np.array([[1.0, 0.8], [0.8, 0.88]])
        kw = dict(ntypes=2, eps=np.array([[1.0, 1.5], [1.5, 0.0]]), sigma=sig, cutoff_list=2.5 * sig)
    params = W.lj_params(box, integrator=integrator, friction=1.0, **kw)
    typ = (rng.random(len(pos)) < 0.2).astype(np.int32) if types == 2 else np.zeros(len(pos), np.int32)
    return pos, W.thermal_velocities(len(pos), 1.44, rng), typ, params


@pytest.mark.parametrize("cells,vacant,types,integrator", [
    ((4, 4, 4), 0, 1, 0), ((4, 4, 4), 227, 1, 0), ((4, 4, 4), 256 - 33, 2, 1), ((5, 4, 6), 3, 2, 0),
    ((9, 7, 8), 1, 1, 1), ((12, 12, 12), 31, 1, 2)])
def test_exchange_equals_full_list(cells, vacant, types, integrator):
    import cavgpu as G

    pos, vel, typ, params = fluid(cells, vacant, types=types, integrator=integrator)
    got = {}
    for tpa in (1, 2, 4, 8):
        s = G.System(pos, vel, typ, params, precision=G.FP64, tpa=tpa)
        s.setup()
        a0, t0 = s.state()[2], s.thermo()
        s.step(12)
        got[tpa] = (a0, *s.state(), np.array([t0["virial"], t0["pe"], s.thermo()["virial"], s.thermo()["pe"]]))
        s.close()
    for tpa in (2, 4):
        for x, y in zip(got[1][:4], got[tpa][:4]):
            np.testing.assert_array_equal(x, y)
    # a sum of ~60 pair terms, each within a few ulp, in another order: |terms| reach 1e3, so
    # 60 * 1e3 * 2^-52 = 1.3e-11 at most on an acceleration; over 12 steps that stays below 1e-10
    assert np.abs(got[1][0] - got[8][0]).max() < 2e-11
    for x, y in zip(got[1][1:4], got[8][1:4]):
        assert np.abs(x - y).max() < 1e-9
    e1, e8 = got[1][4], got[8][4]
    assert np.all(np.abs(e1 - e8) <= 1e-11 * (np.abs(e8) + len(pos)))


def test_rows_outgrow_the_claimed_space():
    import cavgpu as G

    # a capacity of 128 leaves 64 claimed entries per atom; at this density rows hold ~120
    # words, so that some atoms claim more than 64 of them and the list grows
    pos, vel, typ, params = fluid((6, 6, 6), 0, rho=1.35)
    acc = []
    for cap, tpa in ((128, 1), (512, 1), (512, 8)):
        s = G.System(pos, vel, typ, params, precision=G.FP64, tpa=tpa, nbr_capacity=cap)
        s.setup()
        assert s.stats()["max_neighbours"] <= 128 or cap > 128 or s.stats()["capacity"] > 128
        acc.append(s.state()[2])
        s.close()
    np.testing.assert_array_equal(acc[0], acc[1])
    assert np.abs(acc[0] - acc[2]).max() <= 1e-13 * np.abs(acc[2]).max() * 60
