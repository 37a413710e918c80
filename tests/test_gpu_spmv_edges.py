"""Sparse products at the edges of the kernels' tiles against FP64 sums on the
host: row lengths around the groups of four and eight entries (0 to 17, mixed
in a slice), row counts around a slice and a thread block, odd and even numbers
of right-hand sides up to 256, and vectors that are 8- but not 16-byte aligned.
A row's sum has at most 18 terms, so it is off by at most 18 eps of the sum of
the terms' magnitudes."""

import numpy as np
import pytest
import scipy.sparse as sp

from rchol_gb300 import _lib

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    """Symmetric, rows of uneven length: a band and a few long rows."""
    rng = np.random.default_rng(seed)
    A = sp.lil_matrix((n, n))
    for i in range(n):
        for j in range(i + 1, min(n, i + 1 + int(rng.integers(0, 9)))):
            A[i, j] = A[j, i] = -rng.uniform(0.1, 2.0)
    A = A.tocsr()
    A.setdiag(np.asarray(-A.sum(axis=1)).ravel() + 1.0)
    A.sort_indices()
    return A


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 1000])
@pytest.mark.parametrize("k", [1, 2, 3, 7, 8, 32, 33, 255, 256])
def test_spmv_edges(n, k, offset):
    torch = pytest.importorskip("torch")
    A = _matrix(n, n)
    x = np.random.default_rng(k).standard_normal((n, k))
    M = _lib.Matrix.create(A.indptr, A.indices, A.data)
    dx = torch.zeros(n * k + offset, dtype=torch.float64, device="cuda")[offset:]
    dy = torch.full((n * k + offset,), float("nan"), dtype=torch.float64, device="cuda")[offset:]
    dx.copy_(torch.tensor(x.ravel()))
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().rchol_gpu_spmv_d(M.ptr, dx.data_ptr(), dy.data_ptr(), k, st))
    y = dy.cpu().numpy().reshape(n, k)
    bound = 18 * np.finfo(np.float64).eps * (abs(A) @ abs(x))
    assert (abs(y - A @ x) <= bound).all()
