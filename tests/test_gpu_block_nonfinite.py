"""A NaN or an infinity in the right-hand side reaches the rows that depend on
it and no others, although a block's inverse is a dense array: every other row
has the bits that it has without it."""

import numpy as np
import pytest
import scipy.sparse as sp

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu

CASES = {
    "leaves_t64": (lambda: generators.laplace_3d_weighted(31, sigma=1.0, seed=3), 64),  # single thread blocks
    "plane_t8": (lambda: generators.laplace_3d(33), 8),  # clusters of every size
    "wide_t4": (lambda: generators.grid_2d_weighted(300, 29), 4),
}


def _reach(M, start):
    """Rows of the triangular matrix M that depend on entry `start`."""
    hit = np.zeros(M.shape[0], dtype=bool)
    cols, todo = M.tocsc(), [start]
    hit[start] = True
    while todo:
        j = todo.pop()
        new = cols.indices[cols.indptr[j]:cols.indptr[j + 1]]
        new = new[~hit[new]]
        hit[new] = True
        todo.extend(new)
    return hit


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", CASES)
def test_nonfinite_rows(cuda, R, name, precision, k):
    import torch

    make, threads = CASES[name]
    A = make()
    tree = R.Tree.build(A.indptr, A.indices, threads)
    F = R.Factor.compute(R.Matrix.create(A.indptr, A.indices, A.data, tree), tree, seed=5, precision=precision)
    assert F.blocked()
    rp, ci, v = F.export()
    U = sp.csr_matrix((v, ci, rp))
    n = U.shape[0]
    lib, st = _lib.lib(), torch.cuda.current_stream().cuda_stream

    def solve(b, transpose):
        x = torch.empty_like(b)
        _lib.check(lib.rchol_gpu_trsv_d(F.ptr, transpose, b.data_ptr(), x.data_ptr(), k, st))
        return x

    b = torch.tensor(np.random.default_rng(1).standard_normal((n, k)), device=cuda)
    for transpose, M in ((0, U.T.tocsr()), (1, U)):
        x = solve(b, transpose)
        for at in (0, 1, n // 3, n // 2, n - 40, n - 1):
            rows = torch.tensor(_reach(M, at), device=cuda)
            for bad in (float("nan"), float("inf")):
                c = b.clone()
                c[at, k - 1] = bad
                y = solve(c, transpose)
                assert torch.equal(y[:, : k - 1], x[:, : k - 1])
                assert torch.equal(y[~rows, k - 1], x[~rows, k - 1]), (transpose, at, bad)
                assert not bool(y[at, k - 1].isfinite())
                if precision == 0:  # in FP32 an entry of an inverse may have rounded to zero
                    assert not bool(y[rows, k - 1].isfinite().any()), (transpose, at, bad)
    _lib.check(lib.rchol_gpu_solve_status(st))
