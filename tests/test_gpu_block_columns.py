"""Several right-hand sides on the block plan (csrc/blocks.cu) against plain
substitution in FP64: both directions and the preconditioner, numbers of
columns around the change of plan (4, 5) and of traversal (32, 33), one column
of a larger array, row counts around the 64 of the column moves, cluster and
single-thread-block stages.  The factors are M-matrices, so nothing cancels;
64 eps per solve is far above what independent roundings give."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu

TOL = {0: 64 * np.finfo(np.float64).eps, 1: 64 * np.finfo(np.float32).eps}
CASES = {
    "one_row": (lambda: generators.laplace_3d(1), 1),
    "64_rows": (lambda: generators.laplace_3d(4), 2),
    "weighted_t16": (lambda: generators.laplace_3d_weighted(17, sigma=1.0, seed=3), 16),
    "grid_t8": (lambda: generators.grid_2d_weighted(63, 65, "loguniform", shift=1e-4, dirichlet=False), 8),
    "grid_t1": (lambda: generators.grid_2d_weighted(131, 133), 1),  # one node in two pieces
}


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", CASES)
def test_block_columns(cuda, R, name, precision):
    import torch

    make, threads = CASES[name]
    A = make()
    tree = R.Tree.build(A.indptr, A.indices, threads)
    F = R.Factor.compute(R.Matrix.create(A.indptr, A.indices, A.data, tree), tree, seed=5, precision=precision)
    rp, ci, v = F.export()
    U = sp.csr_matrix((v, ci, rp))
    L = U.T.tocsr()
    lib, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    b = np.random.default_rng(1).standard_normal((U.shape[0], 67))
    y = spl.spsolve_triangular(L, b, lower=True)
    refs = {0: y, 1: spl.spsolve_triangular(U, b, lower=False), 2: spl.spsolve_triangular(U, y, lower=False)}
    for k in (2, 4, 5, 31, 32, 33, 67, 3):  # the plan grows and is used again
        d = torch.tensor(np.ascontiguousarray(b[:, :k]), device="cuda")
        for call, ref in refs.items():
            x = torch.full_like(d, float("nan"))
            if call == 2:
                _lib.check(lib.rchol_gpu_precond_d(F.ptr, d.data_ptr(), x.data_ptr(), k, st))
            else:
                _lib.check(lib.rchol_gpu_trsv_d(F.ptr, call, d.data_ptr(), x.data_ptr(), k, st))
            _lib.check(lib.rchol_gpu_solve_status(st))
            err = np.linalg.norm(x.cpu().numpy() - ref[:, :k], axis=0) / np.linalg.norm(ref[:, :k], axis=0)
            assert (err <= (2 if call == 2 else 1) * TOL[precision]).all(), (k, call, err.max())
