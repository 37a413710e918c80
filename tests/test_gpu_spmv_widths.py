"""Sparse products for the numbers of right-hand sides around the change of
kernel (a warp per row where at least 7 of 8 lanes have a column) and around
full warps of the other one, on rows of uneven and of equal length, in rounds
of eight entries; against FP64 sums on the host.  A row's sum has at most 18
terms, so it is off by at most 18 eps of the sum of the terms' magnitudes."""

import numpy as np
import pytest
import scipy.sparse as sp

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu


def _uneven(n):
    rng = np.random.default_rng(n)
    i, j = np.nonzero(np.triu(rng.uniform(size=(n, n)) < 8.0 / n, 1))
    W = sp.coo_matrix((-rng.uniform(0.1, 2.0, len(i)), (i, j)), shape=(n, n)).tocsr()
    A = (W + W.T).tocsr()
    A = (A + sp.diags(1.0 - np.asarray(A.sum(axis=1)).ravel())).tocsr()
    keep = np.diff(A.indptr) <= 18  # longer rows lose their off-diagonal entries
    A = (sp.diags(keep.astype(float)) @ A @ sp.diags(keep.astype(float)) + sp.eye(n)).tocsr()
    A.eliminate_zeros()
    A.sort_indices()
    return A


MATRICES = {"uneven": lambda: _uneven(700), "grid2d": lambda: generators.grid_2d_weighted(37, 19),
            "grid3d": lambda: generators.laplace_3d(9)}


@pytest.mark.parametrize("name", MATRICES)
def test_spmv_widths(cuda, name):
    import torch

    A = MATRICES[name]()
    n = A.shape[0]
    M = _lib.Matrix.create(A.indptr, A.indices, A.data)
    st = torch.cuda.current_stream().cuda_stream
    for k in (1, 4, 12, 20, 27, 28, 31, 32, 40, 55, 56, 64, 100, 111, 112, 129, 200, 223, 224, 255, 256):
        x = np.random.default_rng(k).standard_normal((n, k))
        dx = torch.tensor(x, device=cuda)
        dy = torch.full((n, k), float("nan"), dtype=torch.float64, device=cuda)
        _lib.check(_lib.lib().rchol_gpu_spmv_d(M.ptr, dx.data_ptr(), dy.data_ptr(), k, st))
        bound = 18 * np.finfo(np.float64).eps * (abs(A) @ abs(x))
        assert (abs(dy.cpu().numpy() - A @ x) <= bound).all(), k
