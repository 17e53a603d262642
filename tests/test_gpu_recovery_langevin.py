"""Records of a Langevin run whose list overflows at a recorded step.

The temperature of a Langevin step is taken at mid-step, before the list is rebuilt; a step
that halts because its rebuild overflowed is completed by the host, which then folds the
record from the sums the halted step left.  The records must equal those of a run whose
list never overflowed, whichever of a chunk's records the overflow falls on: the run
starts after 0, 1 and 2 steps, so that each record period meets it at different places.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("every", [1, 3])
@pytest.mark.parametrize("first", [0, 1, 2])
def test_langevin_records_of_an_overflowed_step(precision, every, first):
    pos, vel, typ, p = W.lj_fluid((10, 10, 10), rho=0.65, temperature=1.44, seed=2024)
    p = dict(p, integrator=G.VELOCITY_VERLET_LANGEVIN, lang_temperature=1.44, lang_friction=1.0, seed=77, n_r_df=0)
    runs = {}
    for cap in (64, 512):
        s = G.System(pos, vel, typ, p, precision=precision, nbr_capacity=cap)
        s.setup()
        if first:
            s.step(first)
        th = s.run(300, every)
        runs[cap] = (th, s.stats(), s.state(), s.thermo())
        s.close()
    assert runs[64][1]["capacity"] > 64 and runs[512][1]["capacity"] == 512  # only the small list overflowed
    np.testing.assert_array_equal(runs[64][0], runs[512][0])
    for a, b in zip(runs[64][2], runs[512][2]):
        np.testing.assert_array_equal(a, b)
    assert runs[64][3] == runs[512][3]
