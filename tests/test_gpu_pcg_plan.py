"""PCG applies the preconditioner by the record streams (csrc/trsv.cu) for
factors of both precisions, whatever plan rchol_gpu_trsv_d and
rchol_gpu_precond_d take: CG amplifies rounding, so the order of the
preconditioner's sums is part of what a solve returns.  Iterates and counts of
a factor as it comes equal, bit for bit, those of the same factor held to the
record streams by RCHOL_TRSV_FORMAT=1 (the formats that are chosen without it)."""

import numpy as np
import pytest

from rchol_gb300 import autograd, generators

pytestmark = pytest.mark.gpu


def _both(monkeypatch, make):
    own = make()
    monkeypatch.setenv("RCHOL_TRSV_FORMAT", "1")
    streams = make()
    monkeypatch.delenv("RCHOL_TRSV_FORMAT")
    return own, streams


GRIDS = {
    "cube_t32": (lambda: generators.laplace_3d_weighted(24, sigma=1.0, seed=3), 32),
    "plane_t1": (lambda: generators.grid_2d_weighted(130, 97, "loguniform", shift=1e-4, dirichlet=False), 1),
}


@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("grid", GRIDS)
def test_pcg(cuda, R, monkeypatch, grid, precision, k):
    make, threads = GRIDS[grid]
    A = make()
    tree = R.Tree.build(A.indptr, A.indices, threads)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    own, streams = _both(monkeypatch, lambda: R.Factor.compute(Ad, tree, seed=5, precision=precision))
    b = np.random.default_rng(1).standard_normal((A.shape[0], k))
    x, relres, itr = R._pcg_host(Ad, own, b, 1e-10, 200)
    xs, relres_s, itr_s = R._pcg_host(Ad, streams, b, 1e-10, 200)
    assert np.array_equal(itr, itr_s) and np.array_equal(x, xs) and np.array_equal(relres, relres_s)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_batch(cuda, R, monkeypatch, precision):
    rng = np.random.default_rng(4)
    mats = [generators.grid_2d_weighted(int(a), int(c), "lognormal", sigma=0.5, rng=rng)
            for a, c in rng.integers(20, 150, size=(15, 2))]
    bs = [rng.standard_normal(A.shape[0]) for A in mats]
    own, streams = _both(monkeypatch, lambda: R.Batch(mats, threads=1, seed=2, precision=precision))
    (xs, relres, itr), (xs_s, relres_s, itr_s) = own.solve(bs), streams.solve(bs)
    assert np.array_equal(itr, itr_s) and np.array_equal(relres, relres_s)
    assert all(np.array_equal(x, y) for x, y in zip(xs, xs_s))


def test_gradient(cuda, R, monkeypatch):
    import torch

    n = 60
    idx = np.arange(n * n).reshape(n, n)
    ei = np.concatenate([idx[:-1].ravel(), idx[:, :-1].ravel()])
    ej = np.concatenate([idx[1:].ravel(), idx[:, 1:].ravel()])
    rng = np.random.default_rng(0)
    w0 = torch.tensor(10.0 ** rng.uniform(-2.0, 2.0, len(ei)), device=cuda)
    b0 = torch.tensor(rng.standard_normal(n * n), device=cuda)

    def solve():  # the forward and the backward pass factor A(w) anew
        op = autograd.LaplacianOperator(n * n, ei, ej, shift=1e-4, nt=4, seed=1)
        w, b = w0.clone().requires_grad_(), b0.clone().requires_grad_()
        x = autograd.laplacian_solve(w, b, op, tol=1e-12)
        x.backward(x.detach())
        return x.detach(), w.grad, b.grad

    assert all(torch.equal(p, q) for p, q in zip(*_both(monkeypatch, solve)))


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_plan_info(cuda, R, monkeypatch, precision):
    """The reported plan is the one PCG applies."""
    A = generators.laplace_3d(24)
    tree = R.Tree.build(A.indptr, A.indices, 16)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    own, streams = _both(monkeypatch, lambda: R.Factor.compute(Ad, tree, seed=5, precision=precision))
    for transpose in (False, True):
        assert own.plan_info(transpose) == streams.plan_info(transpose)
