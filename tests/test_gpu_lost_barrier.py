"""A grid barrier whose bounded wait runs out: an error status, and no later launch on the same
control record waits on the barrier or uses what it guards (lost_barrier.cu)."""
import os
import subprocess

import pytest

import abm_b200

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "biofilm-abms_b200")


def test_lost_barrier_stops_the_context(tmp_path):
    lib = os.path.join(os.path.dirname(os.path.abspath(abm_b200.__file__)), "_lib")
    exe = os.fspath(tmp_path / "lost_barrier")
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                           "-I", os.path.join(PKG, "csrc"), "-o", exe, os.path.join(HERE, "lost_barrier.cu"),
                           "-L", lib, "-l:libabm_b200.so", "-Xlinker", "-rpath", "-Xlinker", lib])
    done = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr
    assert done.stdout.strip() == "ok"
