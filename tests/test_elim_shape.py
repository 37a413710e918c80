"""Shapes of the elimination per tree depth (csrc/elim_shape.hpp, CPU): a wide
column enlarges the buffers of its own depth only, and every depth's buffers
fit where the shape puts them."""

import os
import subprocess

import pytest

from conftest import ROOT

SMEM, SMS = 227 * 1024, 152


@pytest.fixture(scope="module")
def shapes():
    scratch = os.path.join(ROOT, "tests", ".scratch")
    os.makedirs(scratch, exist_ok=True)
    exe = os.path.join(scratch, "elim_shape")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "rchol_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "elim_shape.cpp"), "-o", exe], check=True)

    def run(depths):
        args = [str(SMEM), str(SMS)] + [str(v) for d, t in enumerate(depths) for v in (d + 1, *t)]
        out = subprocess.run([exe, *args], check=True, capture_output=True, text=True).stdout.split("\n")
        return [tuple(int(v) for v in line.split()) for line in out if line]

    return run


def test_wide_root_column_leaves_other_depths_alone(shapes):
    plain = [(4, 1024, 0, 1), (4, 768, 0, 2), (4, 48, 0, 1024)]  # initial degree, slab, widest misfit, nodes
    for widest in (1500, 2049, 3000, 4097, 9000, 100000):
        hub = [(4, 1024, widest, 1), *plain[1:]]
        assert shapes(hub)[1:] == shapes(plain)[1:], widest
        assert shapes(hub)[0][1] >= widest


@pytest.mark.parametrize("nodes", [1, 1216, 1217, 100000])
@pytest.mark.parametrize("width", [1, 33, 256, 257, 2048, 2049, 4096, 4097, 5700, 8193])
def test_buffers_fit(shapes, width, nodes):
    (four, emax, node_smem, per_block), = shapes([(0, 0, width, nodes)])
    assert emax >= width and emax & (emax - 1) == 0
    assert bool(four) == (nodes <= 8 * SMS and max(256, emax) * 96 <= SMEM - 2048)
    assert node_smem == (emax * (96 if four else 40) if four or emax * 40 <= SMEM else 0)
    assert node_smem * per_block + (2048 if four else 0) <= SMEM and per_block in ((1,) if four else (1, 2, 3, 4))
