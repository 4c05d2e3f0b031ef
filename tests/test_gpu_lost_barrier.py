"""Launches whose blocks wait for one another, when they cannot.  A grid barrier whose bounded
wait runs out: an error status, and no later launch on the same control record waits on the
barrier or uses what it guards (lost_barrier.cu).  A launch that the runtime refuses: the
wrapper says so (refused_launch.cu)."""
import os
import subprocess

import pytest

import abm_b200

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "biofilm-abms_b200")


def run(name, tmp_path):
    lib = os.path.join(os.path.dirname(os.path.abspath(abm_b200.__file__)), "_lib")
    exe = os.fspath(tmp_path / name)
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                           "-I", os.path.join(PKG, "csrc"), "-o", exe, os.path.join(HERE, name + ".cu"),
                           "-L", lib, "-l:libabm_b200.so", "-Xlinker", "-rpath", "-Xlinker", lib])
    done = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr
    return done.stdout.strip()


def test_lost_barrier_stops_the_context(tmp_path):
    assert run("lost_barrier", tmp_path) == "ok"


def test_refused_launch_is_reported(tmp_path):
    assert run("refused_launch", tmp_path) == "cudaErrorCooperativeLaunchTooLarge 0 0"
