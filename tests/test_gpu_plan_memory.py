"""Which plan trsv and precond take belongs to the problem, not to the memory
that happens to be free when the factor is made; and a factor that the record
streams alone have room for is made, whatever the block plan would need."""

import numpy as np
import pytest

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _solve(torch, F, b):
    x = torch.empty_like(b)
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().rchol_gpu_trsv_d(F.ptr, 0, b.data_ptr(), x.data_ptr(), 1, st))
    _lib.check(_lib.lib().rchol_gpu_solve_status(st))
    return x


def _fill(torch, left):
    """Takes all device memory but `left` bytes."""
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(max(0, free - left) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def problem(cuda, R):
    import torch

    A = generators.laplace_3d(50)
    tree = R.Tree.build(A.indptr, A.indices, 32)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    b = torch.tensor(np.random.default_rng(0).standard_normal(A.shape[0]), device=cuda)
    return tree, Ad, b


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_plan_does_not_follow_free_memory(R, problem, precision):
    import torch

    tree, Ad, b = problem
    F = R.Factor.compute(Ad, tree, seed=1, precision=precision)
    x = _solve(torch, F, b)
    del F
    filler = _fill(torch, 640 * MB)
    try:
        F = R.Factor.compute(Ad, tree, seed=1, precision=precision)
        y = _solve(torch, F, b)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert torch.equal(x, y)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_factor_is_made_where_the_streams_fit(R, problem, monkeypatch, precision):
    import torch

    tree, Ad, b = problem
    F = R.Factor.compute(Ad, tree, seed=1, precision=precision)
    x = _solve(torch, F, b)
    del F
    eps = np.finfo(np.float32 if precision else np.float64).eps
    made = {True: 0, False: 0}
    for left in range(400, 112, -16):
        fits = {}
        for streams_only in (True, False):
            if streams_only:
                monkeypatch.setenv("RCHOL_TRSV_FORMAT", "1")
            else:
                monkeypatch.delenv("RCHOL_TRSV_FORMAT", raising=False)
            filler = _fill(torch, left * MB)
            F = None
            try:
                F = R.Factor.compute(Ad, tree, seed=1, precision=precision)
            except R.RcholError as e:
                assert e.status == _lib.ERR_NOMEM
            finally:
                del filler
                torch.cuda.empty_cache()
            fits[streams_only] = F is not None
            if F:
                y = _solve(torch, F, b)
                assert float((x - y).norm()) <= 64 * eps * float(x.norm())
                del F, y
            made[streams_only] += fits[streams_only]
        assert fits[False] or not fits[True], left
        if not fits[True]:
            break
    assert made[True] and made[False]


def test_call_after_one_without_memory(R, problem):
    """A factor that could not be made leaves nothing behind that fails the
    next call."""
    import torch

    tree, Ad, b = problem
    filler = _fill(torch, 32 * MB)
    try:
        with pytest.raises(R.RcholError) as e:
            R.Factor.compute(Ad, tree, seed=1)
        assert e.value.status == _lib.ERR_NOMEM
    finally:
        del filler
        torch.cuda.empty_cache()
    F = R.Factor.compute(Ad, tree, seed=1)
    assert bool(_solve(torch, F, b).isfinite().all())
