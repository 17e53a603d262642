"""The library's host side when device memory runs short or a kernel gives up, without a GPU.

tests/cpp/host_memory.cu drives the C ABI with a stand-in for the CUDA runtime
(tests/cpp/fake_cudart.cpp) whose memory has a limit and whose kernels do not run.
"""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def program():
    sys.path.insert(0, PKG)
    import build as B

    if not os.path.exists(B.LIB):
        B.build()
    out = os.path.join(ROOT, "tests", "cpp", "_build")
    os.makedirs(out, exist_ok=True)
    exe, src = os.path.join(out, "host_memory"), os.path.join(ROOT, "tests", "cpp")
    objs = [os.path.join(B.OBJ, os.path.splitext(s)[0] + ".o") for s in B.SOURCES]
    subprocess.run([B.NVCC, *B.ARCH, "-std=c++17", "-O1", "-cudart", "none", "-I" + os.path.join(ROOT, "include"),
                    "-I" + B.CSRC, "-I" + src, os.path.join(src, "host_memory.cu"), os.path.join(src, "fake_cudart.cpp"),
                    *objs, "-o", exe], check=True, capture_output=True, text=True)

    def run(scenario):
        r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr
        return {k: int(v) for k, v in (line.split() for line in r.stdout.splitlines())}

    return run


def test_step_kernel_stops_when_the_exchange_arrays_do_not_fit_any_more(program):
    """A list that grows in mid-run may leave no room for the pair exchange; the run then goes on
    with kernels over the full list."""
    r = program("exchange_lost")
    assert r["setup"] == 0 and r["run"] == 0
    assert r["steps"] == 400 and r["capacity"] == 320
    assert r["nulls"] == 0  # no step kernel without its arrays
    assert 1 <= r["chunks"] <= 2 and r["graphs"] >= 1


def test_a_growing_list_takes_the_room_of_the_exchange_arrays(program):
    """The list's new rows fit once the arrays that the force can do without are given back."""
    r = program("list_grows")
    assert r["setup"] == 0 and r["run"] == 0
    assert r["steps"] == 400 and r["capacity"] == 320 and r["nulls"] == 0


def test_a_context_takes_the_exchange_arrays_of_an_idle_one(program):
    r = program("second_context")
    assert r["setup"] == 0 and r["run"] == 0 and r["exchange_before"] == 1
    assert r["second_setup"] == 0 and r["second_run"] == 0 and r["exchange_after"] == 0
    assert r["run_again"] == 0 and r["run_last"] == 0 and r["nulls"] == 0


def test_a_context_in_a_call_keeps_its_exchange_arrays(program):
    r = program("busy_context")
    assert r["setup"] == 0 and r["run"] == 0
    assert r["second_setup"] == -6  # CAVGPU_E_NOMEM
    assert r["exchange"] == 1 and r["nulls"] == 0


def test_autotune_takes_the_room_of_its_own_exchange_arrays(program):
    r = program("autotune")
    assert r["setup"] == 0 and r["exchange_before"] == 1
    assert r["autotune"] == 0 and r["run"] == 0 and r["nulls"] == 0


def test_a_context_whose_barrier_gave_up_refuses_every_use_of_its_state(program):
    r = program("stall")
    assert r["setup"] == 0
    for call in ("run", "run_again", "forces", "thermo", "download", "setup_again", "autotune", "pairs"):
        assert r[call] == -2, call  # CAVGPU_E_CUDA
    assert r["named"] == 1 and r["stats"] == 0
    assert r["other"] == 0  # other contexts go on


def test_the_step_kernels_grid_fits_the_device_it_runs_on(program):
    """Blocks of a cooperative launch must all be resident: four per multiprocessor here."""
    r = program("devices")
    assert r["second"] <= 10 * 4 < r["first"] <= 152 * 4
    assert r["first_again"] == r["first"]


def test_pinned_memory_is_taken_by_the_first_run(program):
    r = program("pinned")
    assert r["forces"] == 0 and r["run"] == 0
    assert r["before"] == 0 and r["after"] == 1
