"""Batched PCG, whose warps read 24 rows of 256 chains at a time (6144 rows):
system sizes at and just off that, 256, fewer rows than chains
between them, and several rounds, against the oracle's PCG on each system.  Both sides stop at the same relative residual, in
sums that round differently, so the counts may differ by one where a residual
lies within rounding of the line; the reported residual is the true one to
1e-10 (tol = 1e-8 and sums of at most 13200 terms)."""

import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from conftest import csr_u64
from rchol_gb300 import generators

SIDES = [(96, 64), (3, 2), (83, 74), (58, 106), (2, 2), (16, 16), (120, 110)]  # 6144, 6, 6142, 6148, 4, 256, 13200 rows


@pytest.mark.gpu
def test_batch_pcg_chains(cuda, R, O):
    rng = np.random.default_rng(5)
    mats = [generators.grid_2d_weighted(nx, ny, "lognormal", sigma=0.5, rng=rng) for nx, ny in SIDES]
    sizes = [A.shape[0] for A in mats]
    ptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    U = sp.block_diag(mats, format="csr")
    U.sort_indices()
    T = R.Tree.build_batch(ptr, U.indptr, U.indices, 2)
    perm, part = T.arrays()
    Up = O.reorder(csr_u64(U), perm.astype(np.uint64))
    G, d, _ = O.factor(O.extend(Up), part.astype(np.uint64), oracle.MODE_REF, 11)
    B = R.Batch(mats, threads=2, precision=0, G=G)
    assert np.array_equal(B.perm, perm)
    bs = [rng.standard_normal(m) for m in sizes]
    tol = 1e-8
    Gm = sp.csr_matrix((G[2], G[1].astype(np.int64), G[0].astype(np.int64)))
    Upm = sp.csr_matrix((Up[2], Up[1].astype(np.int64), Up[0].astype(np.int64)))
    bperm = np.concatenate(bs)[perm]
    xs, relres, itr = B.solve(bs, tol=tol, maxit=200)
    again = B.solve(bs, tol=tol, maxit=200)
    for s, A in enumerate(mats):
        a, b = ptr[s], ptr[s + 1]
        _, _, ito = O.pcg(csr_u64(Upm[a:b, a:b].tocsr()), bperm[a:b].copy(), tol, 200, csr_u64(Gm[a:b, a:b].tocsr()))
        assert abs(int(itr[s]) - ito) <= 1, s
        true = np.linalg.norm(A @ xs[s] - bs[s]) / np.linalg.norm(bs[s])
        assert abs(true - relres[s]) <= 1e-10, s
        assert relres[s] <= 1.01 * tol, s
        assert np.array_equal(xs[s], again[0][s]), s  # fixed trees: deterministic
