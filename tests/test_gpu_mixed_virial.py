"""The mixed form's distances carry no common scale error.

Distances are integers times the length of a unit, which an FP32 pair hi + lo holds; if lo
is lost in rounding, every distance of a system is off by up to half an ulp of hi, 2^-25,
and the sum of the pair virials, ~12 times as sensitive, by up to 12 * 2^-25 = 3.6e-7 of
the sum of their magnitudes, always in one direction.  Without it the errors left are those
of single pairs, which average out over 10^5 of them, and of the reciprocal (1 ulp, not
biased by much): below 1e-7 of that sum.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


# box edges 16.8, 21.8, 23.5 and 33.6: their units lose 1e-8 to 3e-8 when hi stands alone
@pytest.mark.parametrize("cells", [10, 13, 14, 20])
@pytest.mark.parametrize("tpa", [1, 4])
def test_virial_and_energy_against_64_bits(cells, tpa):
    rng = np.random.default_rng(cells)
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.12, 0.12, size=pos.shape), box)
    pos[pos >= box] = 0.0
    p = W.lj_params(box)
    s = G.System(pos, np.zeros_like(pos), np.zeros(len(pos), np.int32), p, precision=G.MIXED, tpa=tpa)
    s.setup()
    rows, got = s.pairs(), s.thermo()
    s.close()
    d = pos[rows[:, 1]] + rows[:, 2:] * box - pos[rows[:, 0]]
    u = 1.0 / (d ** 2).sum(1)
    u = u[u >= 1.0 / 2.5 ** 2]
    c3 = 2.5 ** -6.0
    gc, uc = 4.0 * c3 * (6.0 - 12.0 * c3) / 6.25, 4.0 * (c3 * c3 - c3)
    coef = 4.0 * u ** 3 * (6.0 - 12.0 * u ** 3) * u - gc
    w = -coef / u
    e = 4.0 * (u ** 6 - u ** 3) - uc - 0.5 * gc * (1.0 / u - 6.25)
    assert abs(got["virial"] - 0.5 * w.sum()) <= 1e-7 * 0.5 * np.abs(w).sum()
    assert abs(got["pe"] - 0.5 * e.sum()) <= 1e-7 * 0.5 * np.abs(e).sum()
