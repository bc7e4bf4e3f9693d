"""CPU tests of the library's host paths: capi.cu and batched.cu compiled as they
are and linked with a CUDA runtime on the host (host_fake/fake_cuda.cpp) that
remembers its allocations, replays captured launches and makes calls fail."""
import os
import subprocess

import pytest

from conftest import ROOT

FAKE = os.path.join(ROOT, "tests", "host_fake")
CSRC = os.path.join(ROOT, "chllmodel_b200", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    """Builds one of host_fake's programs with the library's sources it names."""
    from chllmodel_b200.build import nvcc

    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    out = tmp_path_factory.mktemp("host_fake")
    # the kernels are not run: no machine code, no optimisation
    flags = ["-gencode", "arch=compute_100a,code=compute_100a", "-O0", "-Xcicc", "-O0",
             "-std=c++17", "--expt-relaxed-constexpr"]

    def obj(path):
        o = out / (os.path.basename(path) + ".o")
        if not o.exists():
            subprocess.run([compiler, *flags, "-c", path, "-o", str(o)], check=True)
        return str(o)

    def build(name, *sources):
        exe = out / os.path.splitext(name)[0]
        objs = [obj(os.path.join(CSRC, s)) for s in sources]
        objs += [obj(os.path.join(FAKE, f)) for f in ("fake_cuda.cpp", name)]
        # launchers of the other sources are not reached
        subprocess.run(["g++", "-o", str(exe), *objs, "-Wl,--unresolved-symbols=ignore-all"],
                       check=True)
        return str(exe)

    return build


def _run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("what", ["larger_map", "tuned", "no_memory", "no_copy"])
def test_batch_launches_only_allocated_memory(program, what):
    _run(program("batch_map.cpp", "batched.cu", "capi.cu"), what)


def test_tuner_and_trials_that_give_up(program):
    _run(program("batch_lost.cpp", "batched.cu", "capi.cu"))


def test_a_wait_that_gave_up_is_reported(program):
    _run(program("lattice_lost.cu", "capi.cu"))


def test_copies_of_a_run_that_fail_are_reported(program):
    _run(program("lattice_lost.cu", "capi.cu"), "copies")


def test_segment_lengths(program):
    _run(program("segments.cu"))


def test_projection_of_the_largest_planes(program):
    _run(program("projection_grid.cpp", "analysis.cu"))
