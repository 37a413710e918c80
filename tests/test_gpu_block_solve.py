"""Triangular solves in large blocks (csrc/blocks.cu) against plain
substitution in FP64: every shape the plan chooses (clusters of 1 to 16 thread
blocks, pieces that end inside a block, one row, nodes longer than a piece),
both directions and precisions, and the factors that must keep the record
streams (mixed signs, rows too dense).  Tolerances: a row's sum has at most m
terms (m = 20,000 here) and the factors are M-matrices, so nothing cancels and
the error is below m eps of the result; 64 eps is far above what independent
roundings give (sqrt(m) eps / 2)."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu

TOL = {0: 64 * np.finfo(np.float64).eps, 1: 64 * np.finfo(np.float32).eps}


def _solve(torch, F, b, transpose):
    d = torch.tensor(b, device="cuda")
    x = torch.empty_like(d)
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().rchol_gpu_trsv_d(F.ptr, transpose, d.data_ptr(), x.data_ptr(),
                                           1 if b.ndim == 1 else b.shape[1], st))
    _lib.check(_lib.lib().rchol_gpu_solve_status(st))
    return x.cpu().numpy()


def _check(torch, F, precision, seed=0):
    rp, ci, v = F.export()
    U = sp.csr_matrix((v, ci, rp))
    L = U.T.tocsr()
    b = np.random.default_rng(seed).standard_normal(U.shape[0])
    for transpose, M, lower in ((0, L, True), (1, U, False)):
        ref = spl.spsolve_triangular(M, b, lower=lower)
        x = _solve(torch, F, b, transpose)
        assert np.linalg.norm(x - ref) <= TOL[precision] * np.linalg.norm(ref), (transpose, precision)


CASES = {
    "one_row": (lambda: generators.laplace_3d(1), 1),
    "7_cubed_t1": (lambda: generators.laplace_3d(7), 1),
    "17_cubed_t2": (lambda: generators.laplace_3d(17), 2),  # a long leaf, one short separator
    "line_t8": (lambda: generators.grid_2d_weighted(1, 5000), 8),  # separators of one row
    "grid_t1": (lambda: generators.grid_2d_weighted(131, 133), 1),  # 17,423 rows: two pieces of one node
    "weighted_t64": (lambda: generators.laplace_3d_weighted(31, sigma=1.0, seed=3), 64),
    "wide_t4": (lambda: generators.grid_2d_weighted(700, 29, "loguniform", shift=1e-4, dirichlet=False), 4),
    "plane_t8": (lambda: generators.laplace_3d(33), 8),  # separators of 1,089 rows: every cluster size
}


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", CASES)
def test_block_solve(cuda, R, name, precision):
    import torch

    make, threads = CASES[name]
    A = make()
    tree = R.Tree.build(A.indptr, A.indices, threads)
    F = R.Factor.compute(R.Matrix.create(A.indptr, A.indices, A.data, tree), tree, seed=5, precision=precision)
    _check(torch, F, precision)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["dense", "random", "mixed_signs"])
def test_factor_from_elsewhere(cuda, R, kind, precision):
    """Factors without a tree: dense rows, scattered entries, and positive
    off-diagonal entries (which rule the large inverses out)."""
    import torch

    rng = np.random.default_rng(2)
    if kind == "dense":
        M = sp.csr_matrix(np.triu(rng.uniform(-1.0, 0.0, (900, 900)), 1) / 900 + np.eye(900))
    else:
        n = 20000
        lo, hi = (-0.2, 0.0) if kind == "random" else (-0.1, 0.1)
        M = (sp.triu(sp.random(n, n, 2e-4, random_state=3, data_rvs=lambda k: rng.uniform(lo, hi, k)), 1)
             + sp.eye(n)).tocsr()
    M.sort_indices()
    _check(torch, R.Factor.from_host(M.indptr, M.indices, M.data, precision=precision), precision)
