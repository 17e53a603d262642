"""The step kernel of small systems (all steps of a chunk in one launch) against the same
steps launched kernel by kernel: states, thermo records and rebuild counts bit for bit.

Sizes from less than a block's worth of atoms to the last one it takes, odd counts, unequal
edges, both lane counts (4 below 24,576 slots, 2 above), every integrator, record periods of
every step, some and none, chunks that do not divide the steps, and replicas.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(cells, vacant, types, integrator, seed=3):
    import workloads as W

    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice(cells, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    pos = pos[np.sort(rng.permutation(len(pos))[vacant:])]
    kw = {}
    if types == 2:
        sig = np.array([[1.0, 0.8], [0.8, 0.88]])
        kw = dict(ntypes=2, eps=np.array([[1.0, 1.5], [1.5, 0.5]]), sigma=sig, cutoff_list=2.5 * sig,
                  mass=np.array([1.0, 2.0]))
    params = W.lj_params(box, integrator=integrator, friction=1.0, seed=9, **kw)
    typ = (rng.random(len(pos)) < 0.2).astype(np.int32) if types == 2 else np.zeros(len(pos), np.int32)
    return pos, W.thermal_velocities(len(pos), 1.44, rng), typ, params


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,vacant,types,integrator,steps,every,spg", [
    ((4, 4, 4), 0, 1, 0, 40, 0, 0), ((4, 4, 4), 256 - 37, 1, 0, 31, 1, 7), ((5, 4, 6), 3, 2, 1, 33, 3, 0),
    ((9, 7, 8), 1, 1, 2, 30, 5, 11), ((13, 11, 9), 17, 2, 0, 61, 0, 25), ((11, 13, 10), 2, 1, 1, 40, 1, 0),
    ((18, 18, 18), 5, 1, 0, 25, 4, 0), ((20, 20, 20), 1, 2, 1, 25, 0, 0)])
def test_step_kernel_equals_single_kernels(precision, cells, vacant, types, integrator, steps, every, spg):
    import cavgpu as G

    pos, vel, typ, params = system(cells, vacant, types, integrator)
    out = []
    for n in (spg, -1):
        s = G.System(pos, vel, typ, params, precision=G.FP64 if precision == "fp64" else G.MIXED, steps_per_graph=n)
        s.setup()
        rec = s.run(steps, every) if every else s.step(steps)
        s.step(1)
        out.append((s.state(), rec, s.thermo(), s.stats()))
        s.close()
    (a, ra, ta, sa), (b, rb, tb, sb) = out
    assert sa["rebuilds"] == sb["rebuilds"] > 1 and sa["steps"] == sb["steps"] == steps + 1
    if precision == "mixed" or len(pos) <= 12288:  # (beyond, the FP64 form runs its steps in graphs)
        assert sa["kernel_launches"] < sb["kernel_launches"] / 4  # a chunk was one launch
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    if every:
        np.testing.assert_array_equal(ra, rb)
    assert ta == tb


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("integrator", [0, 1])
def test_step_kernel_batch(precision, integrator):
    import cavgpu as G

    systems = []
    for r, (cells, vacant) in enumerate([((4, 4, 4), 9), ((5, 5, 5), 0), ((7, 4, 6), 1), ((9, 9, 9), 100)]):
        pos, vel, typ, params = system(cells, vacant, 1, integrator, seed=20 + r)
        systems.append((pos, vel, typ, params["lo"], params["hi"]))
    out = []
    for n in (0, -1):
        s = G.Batch(systems, params, precision=G.FP64 if precision == "fp64" else G.MIXED, steps_per_graph=n)
        s.setup()
        s.step(45)
        out.append((s.state(), s.thermo_batch(), s.stats()))
        s.close()
    (a, ta, sa), (b, tb, sb) = out
    assert sa["rebuilds"] == sb["rebuilds"]
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(ta, tb)
