"""A caller's start block has k + oversampling columns also where the solver
takes the whole Gram of a small mode instead of iterating: it plays no part
there, and no more of it than its own columns is read."""
import numpy as np
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", ["cpu", "cuda"])
def test_start_block_of_a_mode_solved_whole(device):
    dims, k, s = (26, 25, 26), 8, 24
    tree = ht.reference_tree_3d([1, k, k, k, k])
    X = synth.exact_ht(dims, tree, noise_rel=1e-3, seed=3)
    x = torch.from_numpy(np.ascontiguousarray(X.transpose(2, 1, 0))).cuda()
    start = [torch.randn(s, n).t().to(device) for n in dims]
    got = ht.decompose(x, tree, precision="fp32", eig_iters=1, sketch=start)
    want = ht.decompose(x, tree, precision="fp32", eig_iters=1)
    for t in want.U:
        P, Q = got.U[t].double(), want.U[t].double()
        assert (P @ P.t() - Q @ Q.t()).abs().max() < 1e-5   # the same subspace
