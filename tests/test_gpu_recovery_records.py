"""The record of a step that the host completed after its list had overflowed.

The halted step's force and record are done again by themselves; the record must be folded
in the order of an uninterrupted run, so that it equals that run's bit for bit.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("seed", [2024, 2025, 2026, 2027, 2028, 2029])
def test_record_of_an_overflowed_step(precision, seed):
    pos, vel, typ, p = W.lj_fluid((10, 10, 10), rho=0.65, temperature=1.44, seed=seed)
    runs = {}
    for cap in (64, 512):
        s = G.System(pos, vel, typ, p, precision=precision, nbr_capacity=cap)
        s.setup()
        runs[cap] = (s.run(300, 1), s.stats(), s.state())
        s.close()
    assert runs[64][1]["capacity"] > 64 and runs[512][1]["capacity"] == 512  # only the small list overflowed
    np.testing.assert_array_equal(runs[64][0], runs[512][0])
    for a, b in zip(runs[64][2], runs[512][2]):
        np.testing.assert_array_equal(a, b)
