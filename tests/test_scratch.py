"""The library's host code without a GPU, above all the device memory that a mesh
keeps for its solves (queues, packet pools, sums): tests/cpp/scratch_check.cu, linked with the
library's objects in place of the CUDA runtime, runs the entry points and looks
at what they allocate, free and launch."""
import glob
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OBJ = os.path.join(ROOT, "_build", "obj")
CSRC = os.path.join(ROOT, "kratos_polrad_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(
    not os.path.exists(NVCC) or not os.path.exists(os.path.join(OBJ, "kp_walk.o")),
    reason="nvcc or the library's objects missing")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("scratch")
    own = str(d / "scratch_check.o")
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false",
                    "-I", CSRC, "-I", os.path.join(CSRC, "host"), "-I", os.path.join(ROOT, "include"),
                    "-c", os.path.join(ROOT, "tests", "cpp", "scratch_check.cu"), "-o", own], check=True)
    objs = [own, *sorted(glob.glob(os.path.join(OBJ, "*.o")))]
    names = subprocess.run(["nm", "-u", *objs], check=True, capture_output=True, text=True).stdout.split()
    linked = sorted({n for n in names if n.startswith("__cudaRegisterLinkedBinary")})
    exe = str(d / "scratch_check")
    # what is not faked stays unresolved: a call to it ends the program
    subprocess.run(["g++", *objs, *(f"-Wl,--defsym={n}=fake_register" for n in linked),
                    "-Wl,--unresolved-symbols=ignore-all", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["host_mesh", "tape_pool", "captured", "other_capture", "short_memory", "shares", "first_solve", "order_by_count"])
def test_scratch(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == f"OK {what}\n", r.stdout + r.stderr
