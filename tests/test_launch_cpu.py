"""What the library launches, and what it makes of the kernels' reports, on a
CUDA runtime that lives on the host (fake_cudart.h): no GPU and no kernel runs.
The cases are in launch_cases.cpp."""
import os
import subprocess

import pytest

from fortfem_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
OBJECTS = ["kernels_pcg.cu.o", "kernels_pcg_resident.cu.o", "kernels_assemble.cu.o",
           "kernels_ad.cu.o"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    build.build()
    exe = tmp_path_factory.mktemp("launch") / "launch_cases"
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + cuda, "-I" + build.CSRC,
                    "-I" + os.path.join(HERE, "..", "include"),
                    os.path.join(HERE, "launch_cases.cpp"),
                    *[os.path.join(build.BUILD, o) for o in OBJECTS], "-o", str(exe), "-lpthread"],
                   check=True)
    return str(exe)


def run(program, case):
    r = subprocess.run([program, case], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("kernel", ["cluster", "single"])
def test_batch_reports_a_wait_that_ran_out(program, kernel):
    """Of three systems the second's control word says that a CTA other than the
    first gave up: it alone is reported so, and again by the next batch."""
    run(program, "batch_status_" + kernel)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed16", "large"])
def test_group_batch_is_one_launch(program, precision):
    """large: mixed systems that no group of CTAs holds on chip."""
    run(program, "groups_" + precision)


def test_adjoint_beside_another_thread(program):
    """Orders 5 (182 KB of shared memory) and 6 (59 KB) run the same kernel."""
    run(program, "threads_adjoint")


@pytest.mark.parametrize("what", ["p1", "p2", "nedelec", "batch"])
def test_assembly_beside_another_thread(program, what):
    """A thread that assembles a mesh of short columns comes between the calls of
    one with long columns: both launches are accepted."""
    run(program, "threads_" + what)
