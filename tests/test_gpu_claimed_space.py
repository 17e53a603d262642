"""The FP64 pair exchange when its own space, and nothing else, runs out; batches either side
of the step kernel's replica limit.

At a capacity of 128 an atom has room for 64 claimed and 64 received entries.  Rows of at most
124 words (105 to 124 here) fit the list, but some atoms claim or receive more than 64: the list
must grow for those alone.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def dense(seed=11):
    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice((6, 6, 6), 1.22)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape) * (0.8442 / 1.22) ** (1 / 3), box)
    pos[pos >= box] = 0.0
    return pos, W.thermal_velocities(len(pos), 1.0, rng), np.zeros(len(pos), np.int32), W.lj_params(box, dt=0.002)


def test_claims_outgrow_their_space_while_the_rows_fit():
    system, out = dense(), {}
    for cap, tpa in ((128, 1), (128, 4), (512, 1), (128, 8)):
        s = G.System(*system, precision=G.FP64, tpa=tpa, nbr_capacity=cap)
        s.setup()
        a0, st = s.state()[2], s.stats()
        s.step(10)
        out[cap, tpa] = (a0, *s.state())
        assert st["max_neighbours"] <= 128
        # the full list of eight lanes needs no such space
        assert st["capacity"] == (128 if tpa == 8 else cap) if (cap > 128 or tpa == 8) else st["capacity"] > 128
        s.close()
    for other in ((128, 4), (512, 1)):
        for x, y in zip(out[128, 1], out[other]):
            np.testing.assert_array_equal(x, y)
    # sums of ~110 terms of up to 1e3 in another order: 110 * 1e3 * 2^-52, growing over 10 steps
    for x, y in zip(out[128, 1], out[128, 8]):
        assert np.abs(x - y).max() < 1e-9


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("replicas,one_launch", [(6, True), (7, False)])
def test_batches_either_side_of_the_replica_limit(precision, replicas, one_launch):
    systems = [(p, v, np.zeros(len(p), np.int32), np.zeros(3), b)
               for p, v, b, _, _ in W.replica_set(replicas, 200, 700, seed=9)]
    out = []
    for spg in (0, -1):
        s = G.Batch(systems, W.lj_params(systems[0][4]), precision=precision, steps_per_graph=spg)
        s.setup()
        s.step(120)
        if spg == 0:  # chunks of 50 steps; the step kernel leaves a graph of the last step alone
            assert s.stats()["graph_launches"] == (1 if one_launch else 3)
        out.append((*s.state(), s.thermo_batch()))
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
