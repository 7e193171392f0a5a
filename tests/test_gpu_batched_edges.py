"""Grouped batches at the edges of their kernels: leaf blocks on both sides of
the 32- and 64-wide solvers, fibres on both sides of the 256 rows of a
mode-product step and the 512 of an error step, rows of one to nine fibres a
conversion warp, and the ranks where the narrow kernels' widths change.

Against the single-tensor error evaluation in 64 bits; tolerances as in
test_gpu_batched.py.
"""
import pytest

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import synth
from test_gpu_batched import _check_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("k,dims", [
    (1, [(9, 1, 3), (3, 1, 9), (33, 5, 7)]),
    (16, [(16, 16, 17), (15, 17, 31), (64, 8, 65), (73, 7, 64)]),
    (17, [(32, 32, 33), (31, 33, 32), (40, 40, 40), (41, 25, 63)]),
    (24, [(32, 33, 31), (65, 64, 63), (48, 96, 40)]),
    (25, [(33, 32, 34), (90, 70, 50)]),
    (33, [(64, 65, 63), (100, 34, 72)]),
    (64, [(64, 64, 65), (80, 72, 130)]),
])
def test_batch_edges(k, dims, prec):
    pairs = []
    for i, d in enumerate(dims):
        r1, r2 = min(k, d[0]), min(k, d[1])
        r12 = min(k, d[2], r1 * r2)
        tree = ht.reference_tree_3d([1, r12, r12, r1, r2])
        pairs.append((synth.exact_ht(d, tree, noise_rel=1e-3, seed=900 + i), tree))
    assert _check_batch(pairs, prec)["grouped"]
    mixed = [(synth.exact_ht(d, ht.reference_tree_3d([1, 3, 3, 2, 2]), noise_rel=1e-3, seed=950),
              ht.reference_tree_3d([1, 3, 3, 2, 2])) for d in [(44, 20, 12)]]
    _check_batch(mixed + pairs, prec)   # narrow and wide problems in one table
