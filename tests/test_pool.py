"""The scratch pools' host logic over a fake of the CUDA runtime calls."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_scratch_over_a_fake_runtime(tmp_path):
    if not os.path.isfile(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "pool")
    csrc = os.path.join(ROOT, "dendro-gr_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(CUDA, "include"), "-o", exe, os.path.join(ROOT, "tests", "pool", "pool_main.cpp"),
                    "-x", "c++", os.path.join(csrc, "pool.cu"), "-pthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
