"""Launch shapes of the kernels whose CTAs read each other's shared memory, on
the host: split forms carry the cluster dimension alone (a profiler relaunches a
cooperative kernel without it), and a CTA that sees another shape than the one
its arguments were made for refuses it."""
import os
import shutil
import subprocess

from mprgp_gb300 import buildlib

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(buildlib.nvcc()))),
                            "include")


def run_host_test(tmp_path, name):
    exe = str(tmp_path / name)
    cmd = [shutil.which("g++") or "c++", "-std=c++17", "-O1", "-Wall", "-I", buildlib.CSRC, "-I",
           CUDA_INCLUDE, os.path.join(HERE, "cpp", name + ".cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout


def test_split_launch_shapes(tmp_path):
    run_host_test(tmp_path, "test_split_launch")
