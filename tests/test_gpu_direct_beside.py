"""Leaves solved whole beside iterated ones (CTAs of the cooperative eigen-solver
past its barrier) and without any: small modes, sizes up to 64, both ends of the
order of the modes.

Leaf bases against the FP64 oracle's leaf subspaces' energy through the error of
the whole decomposition; tolerances as in test_gpu_batched.py.
"""
import numpy as np
import pytest

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import synth
from test_gpu_batched import TOL, to_dev
import ht_oracle as O

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("k,dims", [(16, (38, 36, 56)), (16, (70, 17, 33)), (8, (90, 9, 130)), (24, (52, 50, 64)),
                                    (20, (26, 150, 64)), (48, (64, 65, 64)), (12, (36, 37, 38)), (3, (3, 70, 5))])
def test_direct_leaves_beside_iterated_ones(k, dims, prec):
    r1, r2 = min(k, dims[0]), min(k, dims[1])
    r12 = min(k, dims[2], r1 * r2)
    tree = ht.reference_tree_3d([1, r12, r12, r1, r2])
    X = synth.exact_ht(dims, tree, noise_rel=1e-3, seed=sum(dims))
    res = ht.decompose(to_dev(X), tree, precision=prec)
    U = {t: a.cpu().numpy().astype(np.float64) for t, a in res.U.items()}
    B = {t: a.cpu().numpy().astype(np.float64) for t, a in res.B.items()}
    Uo, Bo, _ = O.ht_decompose(X, tree)
    assert abs(O.ht_error(X, tree, U, B) - O.ht_error(X, tree, Uo, Bo)) <= TOL[prec]
    for t in tree.leaves():
        assert O.orthogonality_defect(U[t]) < 1e-4
