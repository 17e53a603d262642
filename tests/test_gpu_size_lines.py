"""Either side of the sizes at which a system changes kernels: a warp per atom evaluates the
FP64 pairs up to 6,144 atoms, the step kernel runs FP64 systems of up to 12,288 and mixed ones
of up to 49,151 slots, and four lanes per atom become two after 19,456 slots.  The steps must
equal those launched one kernel at a time, and records (other kernels) be the same as without.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def fluid(n, integrator=0):
    rng = np.random.default_rng(n)
    cells = int(np.ceil((n / 4) ** (1 / 3)))
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    pos = pos[np.sort(rng.permutation(len(pos))[:n])]
    p = W.lj_params(box, integrator=integrator, friction=1.0, seed=3)
    return pos, W.thermal_velocities(n, 1.44, rng), np.zeros(n, np.int32), p


@pytest.mark.parametrize("precision,n,lanes,one_launch", [
    (G.FP64, 6144, 4, True), (G.FP64, 6145, 4, True), (G.FP64, 12288, 4, True), (G.FP64, 12289, 4, False),
    (G.MIXED, 19456, 4, True), (G.MIXED, 19457, 2, True), (G.MIXED, 49151, 2, True), (G.MIXED, 49152, 1, False)])
@pytest.mark.parametrize("integrator", [0, 1])
def test_steps_and_records(precision, n, lanes, one_launch, integrator):
    system, out = fluid(n, integrator), []
    for spg, every in ((0, 4), (-1, 4), (0, 0)):
        s = G.System(*system, precision=precision, steps_per_graph=spg)
        s.setup()
        rec = s.run(24, every) if every else s.step(24)
        st = s.stats()
        assert st["threads_per_atom"] == lanes and st["rebuilds"] > 1
        if spg == 0:
            assert (st["graph_launches"] == 0) == one_launch
        out.append((rec, s.state()))
        s.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for other in out[1:]:
        for x, y in zip(out[0][1], other[1]):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n", [6144, 6145])
@pytest.mark.parametrize("tpa", [1, 2, 4])
def test_pairs_by_atom_equal_pairs_by_task(n, tpa):
    """FP64 forces of recorded steps come from the kernel of a task per warp, others of up to 6,144
    atoms from that of a warp per atom: the same sums for every lane count."""
    system, out = fluid(n), []
    for every in (0, 1):
        s = G.System(*system, tpa=tpa, steps_per_graph=-1)
        s.setup()
        s.run(10, every) if every else s.step(10)
        out.append(s.state())
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
