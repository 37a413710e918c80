"""Factorizations whose columns outgrow their buffers, against the oracle's
device contract bit for bit: the factor must not depend on slab sizes, on the
pool that takes what a slab cannot, or on the runs that are repeated with
larger buffers.

  hub         one column of the root separator with thousands of fill records
              (wider than the four-warp kernel's largest buffer)
  random      a random graph in one node: columns wider than the first
              buffers, and more records past the slabs than the pool holds
  dense_many  more nodes than the four-warp kernel takes (8 per SM), each a
              dense graph: slabs, pool and its exhaustion in the one-warp kernel
"""

import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from conftest import csr_u64

pytestmark = pytest.mark.gpu


def _sddm(n, i, j, w, excess):
    """The Laplacian of the weighted graph plus `excess` on the diagonal."""
    W = sp.coo_matrix((w, (i, j)), shape=(n, n)).tocsr()
    W = W + W.T
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + excess) - W).tocsr()
    A.sort_indices()
    return A


def hub(R):
    rng = np.random.default_rng(1)
    leaf, ring = 7000, 200  # two leaves of independent vertices; the root: the hub, then a ring
    n = 2 * leaf + 1 + ring
    v = np.arange(2 * leaf)
    h, r = 2 * leaf, 2 * leaf + 1 + np.arange(ring)
    i = np.concatenate([v, v, v, r])
    j = np.concatenate([np.full(2 * leaf, h), r[rng.integers(0, ring // 2, 2 * leaf)],
                        r[rng.integers(ring // 2, ring, 2 * leaf)], np.roll(r, 1)])
    A = _sddm(n, np.minimum(i, j), np.maximum(i, j), rng.uniform(0.5, 2.0, len(i)), 1e-2)
    return A, R.Tree.from_partition(np.arange(n), np.array([0, leaf, 2 * leaf, n + 1]))


def random(R):
    rng = np.random.default_rng(2)
    n, m = 5000, 100000
    i, j = rng.integers(0, n, (2, m))
    keep = i != j
    A = _sddm(n, i[keep], j[keep], rng.uniform(0.5, 2.0, int(keep.sum())), 1e-2)
    return A, R.Tree.from_partition(np.arange(n), np.array([0, n + 1]))


def dense_many(R):
    rng = np.random.default_rng(3)
    size, count = 80, 1300
    i, j = np.triu_indices(size, 1)
    A = sp.block_diag([_sddm(size, i, j, rng.uniform(0.5, 2.0, len(i)), 1e-2) for _ in range(count)], format="csr")
    A.sort_indices()
    ptr = np.arange(count + 1, dtype=np.int64) * size
    return A, R.Tree.build_batch(ptr, A.indptr, A.indices, 1)


@pytest.mark.parametrize("case", [hub, random, dense_many], ids=lambda c: c.__name__)
def test_overflow_is_bit_exact(cuda, O, R, case):
    A, tree = case(R)
    F = R.Factor.compute(R.Matrix.create(A.indptr, A.indices, A.data, tree), tree, seed=9)
    perm, part = tree.arrays()
    Ap = O.reorder(csr_u64(A), perm.astype(np.uint64))
    G, d, singular = O.factor(O.extend(Ap), part.astype(np.uint64), oracle.MODE_DEVICE, 9)
    assert not singular
    rp, ci, v = F.export()
    assert np.array_equal(rp, G[0].astype(np.int64))
    assert np.array_equal(ci, G[1].astype(np.int64))
    assert np.array_equal(v, G[2])
    assert np.array_equal(F.pivots(), d[:-1])
