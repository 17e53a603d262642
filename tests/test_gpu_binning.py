"""The list rebuild where its short cuts end, against the oracle.

Atoms are binned in fixed point when they are well inside the box and its grid has at most
65,536 cells along an axis, else in FP64 with the wrap: atoms exactly on faces and cell
boundaries or one ulp beside them, a box of more cells than that, and steps that carry
atoms across faces.  The warps that share a window of small systems keep up to 40 hits
per atom each, else one warp takes the window: a dense solid has more.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CE = 2.8


def face_gas(lengths, n, rng):
    """Atoms at least 0.9 apart, each coordinate with even odds on or an ulp beside a cell boundary."""
    L = np.array(lengths)
    nc = np.floor(L / CE)
    pos = np.empty((0, 3))
    while len(pos) < n:
        k = np.floor(rng.random(3) * np.minimum(nc, 8))
        k = np.where(rng.random(3) < 0.5, k, nc - k)  # near either end of a long box
        edge = k * (L / nc)
        edge = np.choose(rng.integers(0, 3, 3), [np.nextafter(edge, -np.inf), edge, np.nextafter(edge, np.inf)])
        far = (rng.random(3) - 0.5) * np.minimum(L, 24.0)
        p = np.where(rng.random(3) < 0.5, edge, np.mod(far, L))
        p = np.where(p < 0.0, np.nextafter(L, 0.0), np.where(p >= L, 0.0, p))  # lo and the last value below hi
        d = pos - p
        d -= np.round(d / L) * L
        if not len(pos) or (d ** 2).sum(1).min() > 0.81:
            pos = np.vstack([pos, p])
    return pos


def solid():
    import workloads as W

    pos, box = W.fcc_lattice((6, 6, 6), 1.8)  # 175 neighbours within the list cutoff
    pos = np.mod(pos + np.random.default_rng(3).uniform(-0.02, 0.02, pos.shape), box)
    pos[pos >= box] = 0.0
    return pos, box


# 5.7: two cells and a window per axis; 184,000: 65,714 cells
@pytest.mark.parametrize("lengths,n", [((5.7, 5.7, 5.7), 40), ((9.0, 14.1, 8.5), 150), ((184000.0, 9.0, 9.0), 200),
                                       (None, 0)])
def test_rebuild_against_oracle(oracle_lib, lengths, n):
    import cavgpu as G
    import workloads as W

    rng = np.random.default_rng(17)
    pos, box = solid() if lengths is None else (face_gas(lengths, n, rng), np.array(lengths))
    params = W.lj_params(box)
    vel, typ = W.thermal_velocities(len(pos), 1.44, rng), np.zeros(len(pos), np.int32)
    o = oracle_lib.System(pos, vel, typ, params, noise_mode=0)
    o.setup()
    ref, rows = o.state()[2], o.pairs()
    o.step(20)
    xo = o.state()[0]
    # distances carry a few spacings of the longest edge, a pair force of at most ~141 (r = 0.9)
    # changes by 14 times that relatively, an atom has a dozen such neighbours: below 1e3 spacings
    # of a force; over 20 steps (t = 0.1) a position error grows less than tenfold
    ulp = np.spacing(box.max())
    for precision in (G.FP64, G.MIXED):
        s = G.System(pos, vel, typ, params, precision=precision)
        s.setup()
        np.testing.assert_array_equal(s.pairs(), rows)
        a = s.state()[2]
        if precision == G.FP64:
            assert np.abs(a - ref).max() <= 1e3 * ulp * 150
        else:
            assert np.sqrt(((a - ref) ** 2).sum() / (ref ** 2).sum()) < 1e-5  # the mixed form's force bar
        s.step(20)
        x = s.state()[0]
        assert np.all((x >= 0.0 - 0.3) & (x <= box + 0.3))  # wrapped when the list was last built, half a skin since
        d = x - xo
        d -= np.round(d / box) * box
        tol = max(1e-9, 1e3 * ulp) if precision == G.FP64 else 1e-4 * max(1.0, np.sqrt((ref ** 2).mean()) / 100)
        assert np.abs(d).max() <= tol
        s.close()



@pytest.mark.parametrize("shape", ["steps", "forces"])
def test_shared_windows_of_a_batch_equal_single_windows(shape):
    """Replicas whose lists are built by several blocks per window (a batch in steps) and by one
    block or one warp (single systems, the forced build of many windows): the same rows, so the
    same FP64 bits."""
    import cavgpu as G
    import workloads as W

    # 8 replicas take the rebuild kernels in steps; 56 have more windows than a forced build shares
    n, lo, hi, steps = (8, 180, 700, 12) if shape == "steps" else (56, 600, 1500, 0)
    systems = [(p, v, np.zeros(len(p), np.int32), np.zeros(3), b)
               for p, v, b, _, _ in W.replica_set(n, lo, hi, rho_range=(0.7, 1.2), seed=8)]
    params = W.lj_params(systems[0][4])
    b = G.Batch(systems, params, precision=G.FP64)
    b.setup()
    b.step(steps)
    got = [b.split(x) for x in b.state()]
    b.close()
    for r in range(0, n, 1 if steps else 11):
        p = dict(params, lo=systems[r][3], hi=systems[r][4])
        s = G.System(*systems[r][:3], p, precision=G.FP64)
        s.setup()
        s.step(steps)
        for x, y in zip(s.state(), got):
            np.testing.assert_array_equal(x, y[r])
        s.close()
