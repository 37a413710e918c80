"""Shapes of the block solves (csrc/blocks.cu) over the stages that a plan can
have, on the CPU: the thread counts that the kernel's index arithmetic and its
launch bounds ask for, and cluster sizes that the device does not run."""

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
GB300 = (76, 36, 15, 7)


@pytest.fixture(scope="module")
def shapes(built):
    if NVCC is None:
        pytest.skip("nvcc not available")
    scratch = os.path.join(ROOT, "tests", ".scratch")
    os.makedirs(scratch, exist_ok=True)
    exe = os.path.join(scratch, "block_shape")
    src = os.path.join(ROOT, "tests", "block_shape.cu")
    csrc = os.path.join(ROOT, "rchol_gb300", "csrc")
    deps = [src] + [os.path.join(csrc, f) for f in ("blocks.cu", "plan.hpp", "common.hpp", "bulk.hpp")]
    if not os.path.exists(exe) or os.path.getmtime(exe) < max(os.path.getmtime(d) for d in deps):
        subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                        os.path.join(ROOT, "include"), "-I", csrc, "-o", exe, src], check=True, capture_output=True)

    def run(fit):
        out = subprocess.run([exe, *map(str, fit)], check=True, capture_output=True, text=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


@pytest.mark.parametrize("fit", [GB300, (76, 36, 15, 0), (76, 36, 0, 0), (0, 0, 0, 0)], ids=str)
def test_threads(shapes, fit):
    for fp32, _, _, _, _, C, B, nown, gl, nv, threads, most, _ in shapes(fit):
        row_threads, per = nown // 4 * gl, 4 if fp32 else 2
        assert nown * C == B and nown % 4 == 0 and nown // 4 <= 64
        assert gl in (8, 16, 32) and gl >= C  # a lane per thread block that a group sends to
        assert row_threads % 32 == 0 and row_threads == nown * (gl // 4)
        assert nv * gl * per >= B and nv in (1, 2, 4)  # every position of a block has a chunk
        assert threads <= most and (threads - row_threads) % 32 == 0
        if C > 1:
            lanes = (threads - row_threads) // nown
            assert lanes in (1, 2, 4, 8, 16, 32) and lanes * nown == threads - row_threads


def test_cluster_sizes_the_device_runs(shapes):
    whole = {row[:5]: row for row in shapes(GB300)}
    assert {row[5] for row in whole.values()} == {1, 2, 4, 8, 16}
    for i in range(4):
        fit = tuple(f if k < i else 0 for k, f in enumerate(GB300))
        for row in shapes(fit):
            assert row[5] <= 1 << i
            same = whole.get(row[:5])
            if same and row[4] == 0 and same[5] <= 1 << i:
                assert row == same  # the others are as they were
