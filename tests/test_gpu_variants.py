"""Paths that a full-sized GPU does not take by itself, in builds of the library whose limits
are lower: a grid barrier that gives up, FP64 forces without the pair exchange, and contexts
that take the exchange arrays of others.
"""
import os
import subprocess

import numpy as np
import pytest

import cavgpu as G
import workloads as W
from conftest import ROOT

pytestmark = pytest.mark.gpu


def variant(name, source, define):
    """The library with one source compiled under a definition of its own."""
    import build as B

    out = os.path.join(ROOT, "tests", "cpp", "_build")
    os.makedirs(out, exist_ok=True)
    obj, lib = os.path.join(out, name + ".o"), os.path.join(out, f"lib{name}.so")
    objs = [os.path.join(B.OBJ, os.path.splitext(s)[0] + ".o") for s in B.SOURCES if s != source]
    newest = max(os.path.getmtime(f) for f in [*objs, os.path.join(B.OBJ, os.path.splitext(source)[0] + ".o")])
    if not os.path.exists(lib) or os.path.getmtime(lib) < newest:
        subprocess.run([B.NVCC, *B.ARCH, *B.FLAGS, define, "-c", os.path.join(B.CSRC, source), "-o", obj], check=True)
        subprocess.run([B.NVCC, *B.ARCH, "-shared", "-cudart", "static", "-o", lib, obj, *objs], check=True)
    return lib


@pytest.fixture
def load(monkeypatch):
    def f(path):
        monkeypatch.setattr(G, "LIB_PATH", path)
        monkeypatch.setattr(G, "_lib", None)

    return f


def fluid(cells, types=1, integrator=0):
    rng = np.random.default_rng(3)
    pos, box = W.fcc_lattice((cells,) * 3, 0.8442)
    pos = np.mod(pos + rng.uniform(-0.1, 0.1, size=pos.shape), box)
    pos[pos >= box] = 0.0
    kw = {}
    if types == 2:
        sig = np.array([[1.0, 0.8], [0.8, 0.88]])
        kw = dict(ntypes=2, eps=np.array([[1.0, 1.5], [1.5, 0.5]]), sigma=sig, cutoff_list=2.5 * sig)
    p = W.lj_params(box, integrator=integrator, friction=1.0, seed=4, **kw)
    return pos, W.thermal_velocities(len(pos), 1.0, rng), (np.arange(len(pos)) % types).astype(np.int32), p


@pytest.mark.parametrize("precision", [G.FP64, G.MIXED], ids=["fp64", "mixed"])
def test_a_barrier_that_gives_up_is_an_error(precision, load):
    """With a limit of one poll some block gives up at the first barrier and every block leaves;
    the context reports it and is not used again, the GPU is."""
    system = fluid(10)
    load(variant("cavgpu_stall", "cav_chunk.cu", "-DCAV_BARRIER_POLLS=1u"))
    s = G.System(*system, precision=precision)
    s.setup()
    for call in (lambda: s.step(200), lambda: s.step(1), s.forces, s.state, s.thermo):
        with pytest.raises(G.CavError) as e:
            call()
        assert e.value.status == G.E_CUDA and "barrier" in str(e.value)
    s.close()
    single = G.System(*system, precision=precision, steps_per_graph=-1)  # kernels without barriers
    single.setup()
    single.step(5)
    single.close()


@pytest.mark.parametrize("cells,types,integrator", [(4, 1, 0), (9, 2, 1), (12, 1, 2)])
def test_forces_without_the_pair_exchange(cells, types, integrator, load):
    """Where the exchange's arrays do not fit, 1, 2 and 4 lanes run the full-list kernel: the same
    bits for all three, and the exchange's results to rounding (as test_gpu_pair_exchange.py
    holds 8 lanes to)."""
    system, got, normal = fluid(cells, types, integrator), {}, G.LIB_PATH
    full = variant("cavgpu_full", "cav_api.cu", "-DCAV_EXCHANGE_LIMIT=0")
    for lib, tpa in ((normal, 4), (full, 1), (full, 2), (full, 4), (full, 8)):
        load(lib)
        s = G.System(*system, tpa=tpa)
        assert s.pair_exchange() == (lib == normal)
        s.setup()
        a0 = s.state()[2]
        s.step(12)
        got[lib, tpa] = (a0, *s.state())
        s.close()
    ref = got[full, 1]
    for tpa in (2, 4):
        for x, y in zip(ref, got[full, tpa]):
            np.testing.assert_array_equal(x, y)
    for other in (got[normal, 4], got[full, 8]):
        for x, y in zip(ref, other):
            assert np.abs(x - y).max() < 1e-9


@pytest.mark.parametrize("cells,integrator", [(4, 0), (9, 2), (17, 1)])
def test_run_goes_on_after_its_arrays_were_given_back(cells, integrator, load):
    """In a build whose allocations fail at first, a second context takes the first one's exchange
    arrays; the first goes on over the full list it has, to rounding as if nothing had happened."""
    system, out, normal = fluid(cells, 1, integrator), [], G.LIB_PATH
    short = variant("cavgpu_short", "cav_api.cu", "-DCAV_SHORT_OF_MEMORY")
    for lib in (normal, short):
        load(lib)
        a = G.System(*system)
        a.setup()
        a.step(23)
        assert a.pair_exchange()
        b = G.System(*system)
        assert a.pair_exchange() == (lib == normal) and b.pair_exchange()
        rec = a.run(24, 4)
        out.append((rec, *a.state(), a.stats()["rebuilds"]))
        b.setup()
        b.step(5)
        b.close()
        a.step(3)
        a.close()
    assert out[0][4] == out[1][4] > 1
    for x, y in zip(out[0][1:4], out[1][1:4]):
        assert np.abs(x - y).max() < 1e-8  # sums in another order (2e-11) over 24 steps
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-10, atol=1e-8 * len(system[0]))
