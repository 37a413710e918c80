"""A caller's CUDA graph of a solve keeps working while the same factor goes on
to serve calls with more right-hand sides, which need larger workspaces: the
replays give bit for bit what the solve gave when it was captured."""

import numpy as np
import pytest

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [False, True], ids=["blocks", "streams"])
@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
def test_replay_after_wider_calls(cuda, R, monkeypatch, precision, k, streams):
    import torch

    if streams:
        monkeypatch.setenv("RCHOL_TRSV_FORMAT", "1")
    A = generators.laplace_3d(18)
    tree = R.Tree.build(A.indptr, A.indices, 16)
    Ad = R.Matrix.create(A.indptr, A.indices, A.data, tree)
    F = R.Factor.compute(Ad, tree, seed=5, precision=precision)
    assert F.blocked() != streams
    lib, n = _lib.lib(), A.shape[0]
    rng = np.random.default_rng(3)

    def solve(b, x):
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(lib.rchol_gpu_trsv_d(F.ptr, 1, b.data_ptr(), x[0].data_ptr(), b.shape[1], st))
        _lib.check(lib.rchol_gpu_precond_d(F.ptr, b.data_ptr(), x[1].data_ptr(), b.shape[1], st))

    def call(cols):
        b = torch.tensor(rng.standard_normal((n, cols)), device=cuda)
        x = [torch.empty_like(b) for _ in range(2)]
        solve(b, x)
        return b, x

    b, x = call(k)
    torch.cuda.synchronize()
    want = [v.clone() for v in x]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve(b, x)
    for cols in (8, 33):
        call(cols)
        R._pcg_host(Ad, F, rng.standard_normal((n, cols)), 1e-8, 50)
        junk = [torch.full((n * cols,), float("nan"), device=cuda, dtype=torch.float64) for _ in range(8)]
        for v in x:
            v.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(v, w) for v, w in zip(x, want)), cols
        assert all(bool(v.isnan().all()) for v in junk), cols
    _lib.check(lib.rchol_gpu_solve_status(torch.cuda.current_stream().cuda_stream))
