"""A device buffer whose allocation failed is empty (csrc/common.hpp, CPU with
a fake runtime): with its size set and no memory behind it, the next call would
take it for allocated and hand a null pointer to a kernel."""

import os
import subprocess

from conftest import ROOT


def test_failed_allocation_leaves_the_buffer_empty():
    scratch = os.path.join(ROOT, "tests", ".scratch")
    os.makedirs(scratch, exist_ok=True)
    exe = os.path.join(scratch, "devbuf")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "rchol_gb300", "csrc"), "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "devbuf.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout
