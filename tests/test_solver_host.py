"""The solver's host side on the CPU: ls_solver.cu over a runtime of host
memory and queued work (tests/cpp/fake_cuda.h), with failures made by an error
code from the faked call."""
import os
import shutil
import subprocess

import pytest

import lsgb300

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sci-solver_level-set_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = str(tmp_path_factory.mktemp("solver_host"))
    exe = os.path.join(d, "solver_host")
    cmd = [nvcc, "-std=c++17", "-O1", "-cudart", "none", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC,
           os.path.join(ROOT, "tests", "cpp", "solver_host.cu"), os.path.join(ROOT, "tests", "cpp", "fake_cuda.cpp"), os.path.join(CSRC, "ls_solver.cu"),
           os.path.join(CSRC, "ls_layout.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


def _check(program, name):
    r = subprocess.run([program, name], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-4000:]


def test_nothing_in_flight_after_an_error(program):
    _check(program, "errors")


def test_iterations_counted_in_any_order(program):
    _check(program, "iterations")


def test_distances_stay_where_a_run_ends(program):
    _check(program, "restarts")


def test_fim_setting_is_the_callers_or_chosen_by_residency(program):
    _check(program, "settings")


def test_iterations_before_the_loop_do_not_grow_with_its_body(program):
    _check(program, "first_iterations")


def test_default_setting_is_the_librarys_choice():
    # an explicit 5 must be told apart from the default
    assert lsgb300.default_params().fim_ctas_per_sm == 0
