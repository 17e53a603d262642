"""Systems with long list rows: list cutoffs or densities beyond the usual.

Rows of more than 132 words are built by one warp per window, where shared windows would
overflow their parts; rows of more than 200 keep two lanes per atom up to 65,536 slots and the
step kernel to one task per resident warp, rows of more than 600 four lanes up to 38,912;
rows of more than 2,048, whose cells hold thousands of atoms, are not for the step kernel.
"""
import numpy as np
import pytest

import cavgpu as G
import workloads as W

pytestmark = pytest.mark.gpu


def fluid(cells, rc, seed=3):
    rng = np.random.default_rng(seed)
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    p = W.lj_params(box, rc=rc)
    return pos, W.thermal_velocities(len(pos), 1.0, rng), np.zeros(len(pos), np.int32), p


def brute_pairs(pos, L, ce):
    rows = []
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            for sz in (-1, 0, 1):
                s = np.array([sx, sy, sz])
                d = (pos[None] + s * L) - pos[:, None]
                i, j = np.nonzero((d * d).sum(2) < ce * ce)
                keep = (i != j) | bool(s.any())
                rows.append(np.column_stack([i[keep], j[keep], np.tile(s, (keep.sum(), 1))]))
    return G.sort_rows(np.concatenate(rows))


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("rho,voids", [(1.7, 2.5), (1.8, 1.0), (2.6, 1.0)])
def test_dense_lists_against_brute_force(rho, voids, precision):
    """A dense slab beside a void (156 words where it is dense, so that parts of shared windows
    overflow and a warp does the window again) and evenly dense solids (165 and 239 words)."""
    pos, box = W.fcc_lattice((6, 6, 6), rho)
    rng = np.random.default_rng(1)
    pos = np.mod(pos + rng.uniform(-0.02, 0.02, pos.shape), box)
    pos[pos >= box] = 0.0
    L = box * np.array([voids, 1.0, 1.0])
    p = W.lj_params(L)
    s = G.System(pos, np.zeros_like(pos), np.zeros(len(pos), np.int32), p, precision=precision)
    s.setup()
    got = s.pairs()
    assert s.stats()["max_neighbours"] > 133  # more than the parts of a shared window hold
    s.close()
    np.testing.assert_array_equal(got, brute_pairs(pos, L, p["nl_cutoff"] * p["nl_coef"]))


# 10 and 19 cells: the step kernel; 22 cells with rows of 281 words: more tasks than resident warps
@pytest.mark.parametrize("cells,rc,graphs", [(10, 3.5, False), (10, 4.0, False), (19, 4.0, False), (22, 4.0, True),
                                             (22, 3.0, False)])
def test_steps_equal_single_kernels(cells, rc, graphs):
    system, out = fluid(cells, rc), []
    for spg in (0, -1):
        s = G.System(*system, precision=G.MIXED, steps_per_graph=spg)
        s.setup()
        rec = s.run(30, 6)
        out.append((rec, *s.state()))
        if spg == 0:
            assert (s.stats()["graph_launches"] > 0) == graphs
        assert s.stats()["rebuilds"] > 1
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("cells,rc,lanes", [(16, 4.0, 4), (22, 4.0, 2), (24, 2.5, 1), (24, 4.0, 2), (26, 4.0, 1), (19, 6.0, 4),
                                            (22, 6.0, 2)])
def test_default_lanes(cells, rc, lanes):
    s = G.System(*fluid(cells, rc), precision=G.MIXED)
    assert s.stats()["threads_per_atom"] == lanes
    s.close()


@pytest.mark.parametrize("cells,graphs,precision", [(9, False, G.FP64), (11, True, G.FP64), (9, False, G.MIXED)])
def test_cells_of_hundreds_of_atoms(cells, graphs, precision):
    """Particles a fifth of the usual size in a box of two list cutoffs: 2,916 and 5,324 atoms in
    eight cells, rows of ~1,500 and ~2,800 words."""
    rng = np.random.default_rng(3)
    L = np.full(3, 5.7)
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    scale = 5.7 / box[0]
    pos = np.mod((pos + rng.uniform(-0.05, 0.05, size=pos.shape)) * scale, L)
    pos[pos >= 5.7] = 0.0
    p = W.lj_params(L, sigma=np.array([[scale]]), dt=0.0005)
    out = []
    for spg in (0, -1):
        s = G.System(pos, W.thermal_velocities(len(pos), 1.0, np.random.default_rng(1)), np.zeros(len(pos), np.int32), p,
                     precision=precision, steps_per_graph=spg)
        s.setup()
        s.run(6, 3)
        out.append(s.state())
        if spg == 0:
            assert (s.stats()["graph_launches"] > 0) == graphs
        s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
