"""Batches whose systems are all short (up to 4096 rows) are summed and updated
by one thread block per system: four kernels an iteration fewer than longer
systems take, and the same PCG as the oracle's per system.  The counts may
differ by one where a residual lies within rounding of the line."""

import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from conftest import csr_u64
from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu


def _launches(B, iterations):
    lib = _lib.lib()
    bs = [np.random.default_rng(0).standard_normal(m) for m in B.sizes]
    B.solve(bs, tol=0.0, maxit=iterations)
    before = lib.rchol_gpu_launch_count()
    B.solve(bs, tol=0.0, maxit=iterations)
    return lib.rchol_gpu_launch_count() - before


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_kernels_per_iteration(cuda, R, precision):
    def per_iteration(side):
        B = R.Batch([generators.grid_2d_weighted(side, 64, "lognormal", sigma=0.5)], threads=1, precision=precision)
        return (_launches(B, 8) - _launches(B, 4)) // 4

    assert per_iteration(64) == per_iteration(65) - 4  # 4096 and 4160 rows


@pytest.mark.parametrize("sides", [[(2, 1), (3, 2), (16, 16), (17, 16), (64, 64)], [(5, 5), (64, 64), (65, 64)]],
                         ids=["one_block", "chains"])
def test_short_systems(cuda, R, O, sides):
    rng = np.random.default_rng(6)
    mats = [generators.grid_2d_weighted(nx, ny, "lognormal", sigma=0.5, rng=rng) for nx, ny in sides]
    sizes = [A.shape[0] for A in mats]
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    U = sp.block_diag(mats, format="csr")
    U.sort_indices()
    perm, part = R.Tree.build_batch(ptr, U.indptr, U.indices, 1).arrays()
    Up = O.reorder(csr_u64(U), perm.astype(np.uint64))
    G, _, _ = O.factor(O.extend(Up), part.astype(np.uint64), oracle.MODE_REF, 11)
    B = R.Batch(mats, threads=1, precision=0, G=G)
    bs = [rng.standard_normal(m) for m in sizes]
    xs, relres, itr = B.solve(bs, tol=1e-8, maxit=200)
    Gm = sp.csr_matrix((G[2], G[1].astype(np.int64), G[0].astype(np.int64)))
    Upm = sp.csr_matrix((Up[2], Up[1].astype(np.int64), Up[0].astype(np.int64)))
    bperm = np.concatenate(bs)[perm]
    for s, A in enumerate(mats):
        a, b = ptr[s], ptr[s + 1]
        _, _, ito = O.pcg(csr_u64(Upm[a:b, a:b].tocsr()), bperm[a:b].copy(), 1e-8, 200, csr_u64(Gm[a:b, a:b].tocsr()))
        assert abs(int(itr[s]) - ito) <= 1, s
        true = np.linalg.norm(A @ xs[s] - bs[s]) / np.linalg.norm(bs[s])
        assert abs(true - relres[s]) <= 1e-10 and relres[s] <= 1.01e-8, s
