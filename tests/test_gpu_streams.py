"""The record streams (csrc/trsv.cu), which PCG applies and which trsv and
precond fall back to, through the entry points that usually take the block
plan: RCHOL_TRSV_FORMAT=1 holds a factor to them, in the formats that are
chosen without the variable.  Single and k-wide solves of both precisions
against plain substitution in FP64.

Tolerances: a row's sum has at most m terms (m = 20,000 here) and the factors
are M-matrices, so nothing cancels; 64 eps per solve is far above what
independent roundings give (sqrt(m) eps / 2)."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu

TOL = {0: 64 * np.finfo(np.float64).eps, 1: 64 * np.finfo(np.float32).eps}
CASES = {
    "7_cubed_t1": (lambda: generators.laplace_3d(7), 1),
    "weighted_t64": (lambda: generators.laplace_3d_weighted(24, sigma=1.0, seed=3), 64),  # warp format at the bottom
    "plane_t8": (lambda: generators.laplace_3d(26), 8),  # pipeline format at the top
    "grid_t1": (lambda: generators.grid_2d_weighted(131, 133), 1),  # 17,423 rows in one node
}


@pytest.fixture
def streams(monkeypatch):
    monkeypatch.setenv("RCHOL_TRSV_FORMAT", "1")


def _factor(R, name, precision):
    make, threads = CASES[name]
    A = make()
    tree = R.Tree.build(A.indptr, A.indices, threads)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    return Ad, R.Factor.compute(Ad, tree, seed=5, precision=precision)


def _apply(torch, F, call, b):
    lib, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    d = torch.tensor(b, device="cuda")
    x = torch.full_like(d, float("nan"))
    k = 1 if b.ndim == 1 else b.shape[1]
    if call == 2:
        _lib.check(lib.rchol_gpu_precond_d(F.ptr, d.data_ptr(), x.data_ptr(), k, st))
    else:
        _lib.check(lib.rchol_gpu_trsv_d(F.ptr, call, d.data_ptr(), x.data_ptr(), k, st))
    _lib.check(lib.rchol_gpu_solve_status(st))
    return x.cpu().numpy()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", CASES)
def test_solves(cuda, R, streams, name, precision):
    import torch

    _, F = _factor(R, name, precision)
    assert not F.blocked()
    rp, ci, v = F.export()
    U = sp.csr_matrix((v, ci, rp))
    L = U.T.tocsr()
    b = np.random.default_rng(1).standard_normal((U.shape[0], 40))
    y = spl.spsolve_triangular(L, b, lower=True)
    refs = {0: y, 1: spl.spsolve_triangular(U, b, lower=False), 2: spl.spsolve_triangular(U, y, lower=False)}
    for k in (1, 2, 5, 32, 33, 40):
        for call, ref in refs.items():
            x = _apply(torch, F, call, np.ascontiguousarray(b[:, :k]))
            err = np.linalg.norm(x - ref[:, :k], axis=0) / np.linalg.norm(ref[:, :k], axis=0)
            assert (err <= (2 if call == 2 else 1) * TOL[precision]).all(), (k, call, err.max())


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_tuned_choices_keep_the_bits(cuda, R, streams, precision):
    import torch

    _, F = _factor(R, "weighted_t64", precision)
    b = np.random.default_rng(2).standard_normal(24 ** 3)
    before = _apply(torch, F, 2, b)
    info = F.tune()
    assert np.array_equal(_apply(torch, F, 2, b), before)
    assert info["ms_after"] <= info["ms_before"]


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_tuning_changes_no_iterate(cuda, R, precision):
    """The same through PCG on a factor as it comes."""
    Ad, F = _factor(R, "weighted_t64", precision)
    b = np.random.default_rng(3).standard_normal((24 ** 3, 1))
    x, _, itr = R._pcg_host(Ad, F, b, 1e-9, 200)
    F.tune()
    y, _, itr2 = R._pcg_host(Ad, F, b, 1e-9, 200)
    assert itr[0] == itr2[0] and np.array_equal(x, y)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", ["weighted_t64", "plane_t8"])
def test_pcg_columns(cuda, R, name, precision):
    """k right-hand sides in one PCG against one at a time.  Both orders of the
    sums stop at the same relative residual, so the counts may differ by one
    where a residual lies within rounding of the line."""
    Ad, F = _factor(R, name, precision)
    n = F.export()[0].size - 1
    b = np.random.default_rng(4).standard_normal((n, 5))
    X, relres, itr = R._pcg_host(Ad, F, b, 1e-10, 200)
    for j in range(5):
        x, rr, it = R._pcg_host(Ad, F, b[:, j:j + 1], 1e-10, 200)
        assert abs(int(itr[j]) - int(it[0])) <= 1
        assert relres[j] <= 1.01e-10 and rr[0] <= 1.01e-10
        # both within the tolerance of the solution: A's condition times 1e-10
        assert np.linalg.norm(X[:, j] - x[:, 0]) <= 1e-6 * np.linalg.norm(x)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_which_factors_are_blocked(cuda, R, precision):
    """Sampled factors take the block plan; one off-diagonal entry above zero
    or a diagonal below it rules its inverses out."""
    _, F = _factor(R, "7_cubed_t1", precision)
    assert F.blocked()
    rp, ci, v = F.export()
    assert R.Factor.from_host(rp, ci, v, precision=precision).blocked()
    for at, value in ((rp[100] + 1, 1e-3), (rp[100], -2.0), (rp[100] + 1, float("nan"))):
        w = v.copy()
        w[at] = value
        assert not R.Factor.from_host(rp, ci, w, precision=precision).blocked(), (at, value)
    w = v.copy()
    w[rp[100] + 1] = 0.0
    assert R.Factor.from_host(rp, ci, w, precision=precision).blocked()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_many_short_systems(cuda, R, precision):
    """One right-hand side of many short systems stays on the record streams
    (a warp per system), several take the block plan; a tree with long
    separators over as many subdomains takes it for one, too."""
    import torch

    A = generators.grid_2d_weighted(16, 16, "lognormal", sigma=0.5)
    B = R.Batch([A] * 1000, threads=1, precision=precision)
    assert not B.F.blocked(1) and B.F.blocked(2)
    rp, ci, v = B.F.export()
    U = sp.csr_matrix((v, ci, rp))
    b = np.random.default_rng(1).standard_normal((U.shape[0], 2))
    y = spl.spsolve_triangular(U.T.tocsr(), b, lower=True)
    z = spl.spsolve_triangular(U, y, lower=False)
    for k in (1, 2):
        x = _apply(torch, B.F, 2, np.ascontiguousarray(b[:, :k]))
        assert np.linalg.norm(x - z[:, :k]) <= 2 * TOL[precision] * np.linalg.norm(z[:, :k])
    A = generators.laplace_3d(32)
    tree = R.Tree.build(A.indptr, A.indices, 1024)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    assert R.Factor.compute(Ad, tree, precision=precision).blocked(1)
