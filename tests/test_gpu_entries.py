"""Many entries of a 3rd-order tensor: ht.evaluate groups them by the row of the
precontracted matrix (csrc/htops.cu) above a number of entries.  Ranks at the
widths of its kernels, counts at the edges of its sorting and product blocks,
rows without entries, all entries in one row, three trees.

Tolerance: an entry is a sum over x of at most 64 products, then over y of at
most 64, after a precontraction over at most 64 twice: 4 * 64 roundings of 2^-24
of the sum of the terms' magnitudes, 1.6e-5 of it.
"""
import numpy as np
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300._lib import HTError
from test_gpu_htformat import random_factors, to_torch_factors
import ht_oracle as O

pytestmark = pytest.mark.gpu


def check(tree, dims, idx, seed=0, host=False):
    """All entries against calls too small to be grouped, some against the oracle."""
    U, B = random_factors(tree, dims, seed=seed)
    f64 = lambda d: {t: np.asarray(a, np.float64) for t, a in d.items()}
    mag = lambda d: {t: np.abs(a) for t, a in f64(d).items()}
    some = np.unique(np.r_[:200, np.random.default_rng(0).integers(0, len(idx), 1000), len(idx) - 200:len(idx)])
    want, terms = (O.ht_entries(tree, m(U), m(B), idx[some]) for m in (f64, mag))
    Ut, Bt = to_torch_factors(U, B)
    dev = torch.from_numpy(idx).cuda()
    got = ht.evaluate(tree, U, B, dims, idx) if host else ht.evaluate(tree, Ut, Bt, dims, dev).cpu().numpy()
    assert got.shape == (len(idx),) and got.dtype == np.float32
    assert (np.abs(got[some] - want) <= 1.6e-5 * terms + 1e-30).all()
    small = torch.cat([ht.evaluate(tree, Ut, Bt, dims, part) for part in dev.split(8000)]).cpu().numpy()
    assert (np.abs(got - small) <= 3.2e-5 * terms.max()).all()


def draw(dims, count, seed):
    rng = np.random.default_rng(seed)
    return np.stack([rng.integers(0, d, size=count) for d in dims], axis=1).astype(np.int64)


@pytest.mark.parametrize("mk", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
@pytest.mark.parametrize("k", [1, 5, 16, 17, 32, 33, 48, 49, 64])
def test_ranks_and_trees(mk, k):
    dims = (70, 67, 65)
    r = [1, k, k, min(k, 63), max(1, k - 1)]
    check(mk(r), dims, draw(dims, 3000000 // (max(1, k - 2) + 8) + 3, k), seed=k)


@pytest.mark.parametrize("count", [115384, 115385, 14 * 8192 + 699, 15 * 8192 - 1, 15 * 8192 + 1])
def test_counts_at_block_edges(count):
    dims = (300, 41, 1025)
    check(ht.reference_tree_3d([1, 20, 20, 18, 20]), dims, draw(dims, count, count), host=count % 2 == 0)


@pytest.mark.parametrize("rows", ["one", "first_and_last", "sorted", "sparse"])
def test_uneven_rows(rows):
    dims, count = (900, 40, 50), 1 << 17
    idx = draw(dims, count, 5)
    if rows == "one":
        for m in range(2):
            idx[:, m] = 17
    elif rows == "first_and_last":
        idx[:, 0] = np.where(idx[:, 0] % 2 == 0, 0, dims[0] - 1)
    elif rows == "sorted":
        idx = idx[np.lexsort((idx[:, 2], idx[:, 1], idx[:, 0]))]
    else:
        idx[:, 0] = idx[:, 0] // 100 * 100
    check(ht.reference_tree_3d([1, 24, 24, 24, 24]), dims, idx)


def test_outside_index_is_refused():
    dims = (64, 64, 64)
    tree = ht.reference_tree_3d([1, 16, 16, 16, 16])
    U, B = random_factors(tree, dims, seed=1)
    idx = draw(dims, 1 << 18, 2)
    for m, v in ((0, 64), (1, -1), (2, 1 << 40)):
        bad = idx.copy()
        bad[12345, m] = v
        with pytest.raises(HTError, match="outside"):
            ht.evaluate(tree, U, B, dims, bad)
    check(tree, dims, idx)
