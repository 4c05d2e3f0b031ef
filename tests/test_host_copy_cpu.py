"""The threaded device-to-host copy when memory runs out at any of its allocations, the start of
a thread among them (host_copy.cpp, with stand-ins of the CUDA calls; no GPU)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(os.path.dirname(HERE), "biofilm-abms_b200", "csrc")


def test_copy_survives_failed_allocations(tmp_path):
    exe = os.fspath(tmp_path / "host_copy")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", "-I", SRC, "-o", exe,
                           os.path.join(HERE, "host_copy.cpp"), os.path.join(SRC, "abm_host.cpp")])
    done = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, "exit %d: %s%s" % (done.returncode, done.stdout, done.stderr)
    assert done.stdout.strip() == "ok"
