"""The kernels of a solve start before the one ahead of them has ended and wait
for it themselves; what comes before and after them in the stream must still be
ordered.  Solves in a long sequence on changing buffers, straight and as a
replayed graph with copies on both sides, give bit for bit what each gives
alone with the GPU idle."""

import numpy as np
import pytest

from rchol_gb300 import _lib, generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 7])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("grid", ["cube_t32", "plane_t4"])
def test_chain_order(cuda, R, grid, precision, k):
    import torch

    A, threads = {"cube_t32": (generators.laplace_3d(21), 32), "plane_t4": (generators.grid_2d_weighted(90, 71), 4)}[grid]
    tree = R.Tree.build(A.indptr, A.indices, threads)
    F = R.Factor.compute(R.Matrix.create(A.indptr, A.indices, A.data, tree), tree, seed=5, precision=precision)
    lib, n = _lib.lib(), A.shape[0]
    bs = [torch.tensor(np.random.default_rng(i).standard_normal((n, k)), device="cuda") for i in range(6)]
    b, x = torch.empty_like(bs[0]), torch.empty_like(bs[0])

    def solve():
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(lib.rchol_gpu_precond_d(F.ptr, b.data_ptr(), x.data_ptr(), k, st))

    alone = []
    for v in bs:
        b.copy_(v)
        torch.cuda.synchronize()
        solve()
        torch.cuda.synchronize()
        alone.append(x.clone())
    # straight: b is overwritten right behind the solve that reads it
    got = []
    for _ in range(5):
        for v in bs:
            b.copy_(v)
            solve()
            got.append(x.clone())
    torch.cuda.synchronize()
    assert all(torch.equal(g, alone[i % 6]) for i, g in enumerate(got))
    # one graph: copy in, solve, copy out, the result solved again
    src, out, twice = torch.empty_like(b), torch.empty_like(b), torch.empty_like(b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        b.copy_(src)
        solve()
        out.copy_(x)
        b.copy_(x)
        solve()
        twice.copy_(x)
    again = []
    for v in alone:
        b.copy_(v)
        solve()
        again.append(x.clone())
    for i, v in enumerate(bs * 3):
        src.copy_(v)
        graph.replay()
        assert torch.equal(out, alone[i % 6]) and torch.equal(twice, again[i % 6])
    _lib.check(lib.rchol_gpu_solve_status(torch.cuda.current_stream().cuda_stream))
