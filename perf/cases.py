"""What the framework is timed on: its solve path through the public entry
points, from a few thousand unknowns to a few million.

A case names a grid, its coefficients, the number of nested-dissection
subdomains, the precision of G and the call.  The grids are the ones of the
repository's configurations and tests:

  poisson3d     7-point Laplacian with Dirichlet boundary, n^3 unknowns
  lognormal3d   the same graph with edge weights exp(N(0,1)), diagonal + 1e-3
  checker3d     8^3-cell checkerboard of 1 and 1e4
  loguniform2d  5-point grid nx x ny, edge weights 10^U(-2,2), diagonal + 1e-4

and the calls

  spmv      y = A x (k vectors)
  forward, backward, precond   solves with G, G^T and both (k vectors)
  pcg       Solver.solve with device vectors, the whole iteration
  batch     Batch.solve: many 2D grids of uneven size at once, host vectors
  factor    Factor.compute (elimination, assembly, solve plan) and G copied out
  grad      laplacian_solve forward and backward

An ordering depends on the grid alone, so a program keeps it while weights and
right-hand sides change; it is kept here for the life of the process too.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import rchol_gb300 as rc
from rchol_gb300 import _lib, autograd, generators

PRECISION = {"fp64": rc.PREC_FP64, "fp32": rc.PREC_FP32}


def listed():
    return [
        # the smallest call: one preconditioner apply inside somebody's own Krylov loop, all launches and latency
        dict(name="precond_12_fp64", call="precond", grid="poisson3d", n=12, leaves=8, precision="fp64", k=1),
        # the product with A, as any iteration makes it
        dict(name="spmv_128", call="spmv", grid="lognormal3d", n=128, leaves=512, precision="fp32", k=1),
        # the product for a block of right-hand sides on the high-contrast matrix
        dict(name="spmv_80_k8", call="spmv", grid="checker3d", n=80, leaves=128, precision="fp32", k=8),
        # one triangular solve of the fast path, subdomains of 4096 unknowns
        dict(name="forward_128_fp32", call="forward", grid="lognormal3d", n=128, leaves=512, precision="fp32", k=1),
        # the other direction in the accurate precision
        dict(name="backward_64_fp64", call="backward", grid="poisson3d", n=64, leaves=64, precision="fp64", k=1),
        # a 2D graph with ragged sides: short separators, many small subdomains
        dict(name="precond_2d_fp32", call="precond", grid="loguniform2d", n=1000, ny=777, leaves=256, precision="fp32",
             k=1),
        # a block of right-hand sides in one traversal of G
        dict(name="precond_80_fp32_k32", call="precond", grid="poisson3d", n=80, leaves=128, precision="fp32", k=32),
        # the reference's own example: Poisson, b uniform, 1e-10
        dict(name="pcg_64_fp64", call="pcg", grid="poisson3d", n=64, leaves=256, precision="fp64", k=1, tol=1e-10),
        # the mixed-precision solve at 1e-8
        dict(name="pcg_128_fp32", call="pcg", grid="lognormal3d", n=128, leaves=512, precision="fp32", k=1, tol=1e-8),
        # many uneven systems in one solve
        dict(name="batch_40", call="batch", systems=40, lo=32, hi=256, leaves=4, precision="fp32", tol=1e-8),
        # set-up of the preconditioner for new weights on a known ordering
        dict(name="factor_80_fp32", call="factor", grid="lognormal3d", n=80, leaves=128, precision="fp32"),
        # learning edge weights: a solve and its adjoint
        dict(name="grad_400", call="grad", n=400, leaves=64, tol=1e-12),
    ]


def draw(rng):
    call = rng.choice(["precond", "precond", "forward", "backward", "spmv", "pcg", "batch", "factor", "grad"])
    if call == "batch":
        lo = rng.randint(16, 64)
        return dict(call=call, systems=rng.randint(5, 36), lo=lo, hi=rng.randint(lo + 20, 256),
                    leaves=rng.choice([1, 2, 4, 8]), precision=rng.choice(["fp32", "fp64"]), tol=1e-8)
    if call == "grad":
        n = round(math.exp(rng.uniform(math.log(48), math.log(380))))
        return dict(call=call, n=n, leaves=_leaves(n * n, rng), tol=1e-12)
    grid = rng.choice(["poisson3d", "lognormal3d", "checker3d", "loguniform2d"])
    precision = rng.choice(["fp32", "fp64"])
    k = rng.choice([1, 1, 1, 2, 5, 8, 16, 32]) if call != "factor" else 1
    top = 75 if call == "factor" else 64 if call == "pcg" else 60 if k > 1 else 110
    if call == "pcg" and k > 1:
        top = 40
    c = dict(call=call, grid=grid, precision=precision)
    if grid == "loguniform2d":
        size = math.exp(rng.uniform(math.log(2000), math.log(top ** 3)))
        c["n"] = round(math.sqrt(size) * rng.uniform(0.5, 1.5))
        c["ny"] = round(size / c["n"])
        size = c["n"] * c["ny"]
    else:
        c["n"] = round(math.exp(rng.uniform(math.log(11), math.log(top))))
        size = c["n"] ** 3
    c["leaves"] = _leaves(size, rng)
    if call != "factor":
        c["k"] = k
    if call == "pcg":
        c["tol"] = rng.choice([1e-8, 1e-10])
    return c


def _leaves(size, rng):
    """A power of two that leaves each subdomain a few hundred to a few thousand unknowns."""
    return 2 ** max(0, round(math.log2(size / math.exp(rng.uniform(math.log(500), math.log(6000))))))


# ---- inputs ------------------------------------------------------------------


def _matrix(case, seed):
    grid, n = case["grid"], case["n"]
    if grid == "poisson3d":
        return generators.laplace_3d(n)
    if grid == "lognormal3d":
        return generators.laplace_3d_weighted(n, 1.0, 1e-3, seed)
    if grid == "checker3d":
        return generators.checkerboard_3d(n)
    return generators.grid_2d_weighted(n, case["ny"], "loguniform", shift=1e-4, dirichlet=False, seed=seed)


@functools.lru_cache(maxsize=None)
def _ordering(three_d, n, ny, leaves):
    A = generators.laplace_3d(n) if three_d else generators.grid_2d_weighted(n, ny)
    return rc.Tree.build(A.indptr, A.indices, leaves).arrays()


def _ordering_of(case):
    return _ordering(case["grid"] != "loguniform2d", case["n"], case.get("ny", 0), case["leaves"])


def _normal(shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _rhs(case, size, seed):
    k = case.get("k", 1)
    b = _normal((size,) if k == 1 else (size, k), seed)
    return torch.erf(b / math.sqrt(2.0)) if case["grid"] == "poisson3d" else b  # uniform in [-1, 1] for Poisson


def _grids(case, seed):
    """The sides belong to the case, the weights and right-hand sides to the seed."""
    sides = np.random.default_rng(case["systems"]).integers(case["lo"], case["hi"] + 1, size=(case["systems"], 2))
    rng = np.random.default_rng(seed)
    mats = [generators.grid_2d_weighted(int(a), int(b), "lognormal", sigma=0.5, rng=rng) for a, b in sides]
    return mats, [rng.standard_normal(m.shape[0]) for m in mats]


def _edges(n):
    idx = np.arange(n * n, dtype=np.int64).reshape(n, n)
    return (np.concatenate([idx[:-1, :].ravel(), idx[:, :-1].ravel()]),
            np.concatenate([idx[1:, :].ravel(), idx[:, 1:].ravel()]))


def _weights(n, seed):
    m = 2 * n * (n - 1)
    return 10.0 ** np.random.default_rng(seed).uniform(-2.0, 2.0, m)


def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        mats, bs = _grids(case, seed)
        return dict(case=case, solver=rc.Batch(mats, threads=case["leaves"], seed=seed,
                                               precision=PRECISION[case["precision"]]), b=bs)
    if call == "grad":
        n = case["n"]
        ei, ej = _edges(n)
        op = autograd.LaplacianOperator(n * n, ei, ej, shift=1e-4, nt=case["leaves"], seed=seed)
        w = torch.as_tensor(_weights(n, seed), device="cuda")
        op.update(w)
        return dict(case=case, op=op, w=w, b=_normal(n * n, seed), target=_normal(n * n, seed + 1))
    A = _matrix(case, seed)
    perm, part = _ordering_of(case)
    if call in ("spmv", "factor"):
        tree = rc.Tree.from_partition(perm, part)
        state = dict(case=case, seed=seed, tree=tree, A=rc.Matrix.create(A.indptr, A.indices, A.data, tree))
        if call == "factor":  # the caller's arrays for G, with room for any of its sampled patterns
            n, room = A.shape[0], 22 * A.shape[0]
            state["G"] = {"row_ptr": np.zeros(n + 1, np.int64), "col_idx": np.zeros(room, np.int64),
                          "val": np.zeros(room)}
    else:
        state = dict(case=case, solver=rc.Solver(A, case["leaves"], seed=seed, precision=case["precision"], perm=perm,
                                                 part=part))
    if call != "factor":
        state["b"] = _rhs(case, A.shape[0], seed)
        state["x"] = torch.empty_like(state["b"])
    return state


# ---- one pass ----------------------------------------------------------------


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "factor":
        F = rc.Factor.compute(state["A"], state["tree"], seed=state["seed"], precision=PRECISION[case["precision"]])
        G = state["G"]
        if F.nnz > len(G["val"]):
            raise RuntimeError("G has more entries than the arrays for it")
        _lib.check(_lib.lib().rchol_gpu_factor_export(F.ptr, _lib.p64(G["row_ptr"]), _lib.p64(G["col_idx"]),
                                                      _lib.pd(G["val"])))
        return G
    if call == "batch":
        # x and the iteration counts; the last digits of a converged residual are rounding noise
        xs, _, iters = state["solver"].solve(state["b"], tol=case["tol"])
        return {"x": np.concatenate(xs), "iters": iters}
    if call == "pcg":
        x, _, iters = state["solver"].solve(state["b"], tol=case["tol"], return_info=True)
        return {"x": x, "iters": iters}
    if call == "grad":
        w, b = state["w"].clone().requires_grad_(), state["b"].clone().requires_grad_()
        x = autograd.laplacian_solve(w, b, state["op"], tol=case["tol"])
        x.backward(x.detach() - state["target"])
        return {"x": x.detach(), "grad_w": w.grad, "grad_b": b.grad}
    b, x, k = state["b"], state["x"], case["k"]
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    if call == "spmv":
        _lib.check(lib.rchol_gpu_spmv_d(state["A"].ptr, b.data_ptr(), x.data_ptr(), k, stream))
        return x
    G = state["solver"].G.ptr
    if call == "precond":
        _lib.check(lib.rchol_gpu_precond_d(G, b.data_ptr(), x.data_ptr(), k, stream))
    else:
        _lib.check(lib.rchol_gpu_trsv_d(G, int(call == "backward"), b.data_ptr(), x.data_ptr(), k, stream))
    # with an FP32 factor the result carries FP32 accuracy and is kept as such
    return x.float() if case["precision"] == "fp32" else x


# ---- what a pass cannot do without -------------------------------------------


def work(case):
    """Bytes: A as CSR (8-byte values, 4-byte columns, 8-byte row pointers), G
    in its precision, every vector once; a PCG reads A once and G twice per
    iteration.  nnz(G) per unknown and the iteration counts are those that
    these grids have been seen to take."""
    call = case["call"]
    if call == "batch":
        mean = (case["lo"] + case["hi"]) / 2.0
        n, k, per_a, per_g, iters = case["systems"] * mean * mean, 1, 5.0, 7.5, 20
    elif call == "grad":
        n, k, per_a, per_g, iters = case["n"] ** 2, 1, 5.0, 7.5, 100
    else:
        two_d = case["grid"] == "loguniform2d"
        n, k = case["n"] * case["ny"] if two_d else case["n"] ** 3, case.get("k", 1)
        per_a = 5.0 if two_d else 7.0
        per_g = 7.5 if two_d else 4.0 + 0.6 * math.log2(max(8, n))
        iters = 50 if two_d else 26
    vs = 4 if case.get("precision") == "fp32" else 8
    a, g = n * (per_a * 12 + 8), n * (per_g * (vs + 4) + 8)
    vec = 8.0 * n * k
    if call == "spmv":
        return {"bytes": a + 2 * vec, "flops": 2 * n * per_a * k}
    if call in ("forward", "backward"):
        return {"bytes": g + 2 * vec, "flops": 2 * n * per_g * k}
    if call == "precond":
        return {"bytes": 2 * g + 2 * vec, "flops": 4 * n * per_g * k}
    if call == "factor":
        return {"bytes": n * per_a * 6 + n * per_g * 16, "flops": 20.0 * n * per_g}
    return {"bytes": iters * (a + 2 * g + 10 * vec), "flops": iters * n * k * (2 * per_a + 4 * per_g + 12)}


# ---- the same in plain 64-bit torch --------------------------------------------


def _csr_t(A):
    return torch.sparse_csr_tensor(torch.as_tensor(A.indptr.astype(np.int64)),
                                   torch.as_tensor(A.indices.astype(np.int64)), torch.as_tensor(A.data),
                                   size=A.shape, dtype=torch.float64, device="cuda")


def _cg(A, b):
    """A x = b by conjugate gradients with the diagonal, until the residual stops falling."""
    M = _csr_t(A)
    dinv = 1.0 / torch.as_tensor(A.diagonal(), device="cuda")[:, None]
    b = b.reshape(A.shape[0], -1)
    x = torch.zeros_like(b)
    for _ in range(3):  # restarted from the true residual
        r = b - M @ x
        goal = 1e-15 * b.norm(dim=0)
        z = dinv * r
        p, rz = z.clone(), (r * z).sum(0)
        for it in range(20000):
            q = M @ p
            alpha = rz / (p * q).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            z = dinv * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
            if it % 50 == 49 and bool((r.norm(dim=0) <= goal).all()):
                break
    return x


def _poisson(n, b):
    """The Poisson matrix is diagonal in the basis of sines along each axis."""
    i = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
    S = torch.sin(math.pi * i[:, None] * i[None, :] / (n + 1)) * math.sqrt(2.0 / (n + 1))
    lam = 2.0 - 2.0 * torch.cos(math.pi * i / (n + 1))

    def along(v):
        return torch.einsum("ai,bj,ck,ijkr->abcr", S, S, S, v)

    h = along(b.reshape(n, n, n, -1))
    h /= (lam[:, None, None] + lam[None, :, None] + lam[None, None, :])[..., None]
    return along(h).reshape(n ** 3, -1)


def exact(case, seed):
    call = case["call"]
    if call == "factor":
        return None  # a sampled factor: its values have no formula but the sampling itself
    if call == "batch":
        mats, bs = _grids(case, seed)
        xs = [_cg(A, torch.as_tensor(b, device="cuda"))[:, 0] for A, b in zip(mats, bs)]
        return {"x": torch.cat(xs), "iters": None}
    if call == "grad":
        n = case["n"]
        ei, ej = _edges(n)
        w = _weights(n, seed)
        op = autograd.LaplacianOperator(n * n, ei, ej, shift=1e-4, nt=1)  # only its pattern: A(w) as scipy CSR
        A = op.matrix(w)
        x = _cg(A, _normal(n * n, seed))[:, 0]
        lam = _cg(A, x - _normal(n * n, seed + 1))[:, 0]
        i, j = torch.as_tensor(ei, device="cuda"), torch.as_tensor(ej, device="cuda")
        return {"x": x, "grad_w": -(lam[i] - lam[j]) * (x[i] - x[j]), "grad_b": lam}
    A = _matrix(case, seed)
    b = _rhs(case, A.shape[0], seed)
    if call == "pcg":
        x = _poisson(case["n"], b) if case["grid"] == "poisson3d" else _cg(A, b)
        return {"x": x.reshape(b.shape), "iters": None}
    perm, _ = _ordering_of(case)
    if call == "spmv":
        return (_csr_t(A[perm][:, perm]) @ b.reshape(len(perm), -1)).reshape(b.shape)
    # the solves take a factor as their input: its values, solved with torch's own sparse substitution
    state = prepare(case, seed)
    rp, ci, v = (torch.as_tensor(t, device="cuda") for t in state["solver"].G.export())
    n = len(perm)
    U = torch.sparse_csr_tensor(rp, ci, v, size=(n, n), dtype=torch.float64, device="cuda")
    x = b.reshape(n, -1)
    if call in ("precond", "forward"):
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
        L = torch.sparse_coo_tensor(torch.stack([ci, row]), v, size=(n, n)).coalesce().to_sparse_csr()
        x = torch.triangular_solve(x, L, upper=False).solution
    if call in ("precond", "backward"):
        x = torch.triangular_solve(x, U, upper=True).solution
    return x.reshape(b.shape)
