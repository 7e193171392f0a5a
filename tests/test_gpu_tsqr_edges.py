"""TSQR of at most 32 columns on both sides of its 16-column steps, its panels of
64 and 128 rows and its trees, with a zero column and a repeated one.

Tolerance: R^T R against A^T A relative to the columns' norms; Householder
folds of at most 15 panels, 32 reflections each, are backward stable to a small
multiple of 32 * 15 * 2^-24 = 2.9e-5 in the worst case.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("m", [1, 63, 64, 65, 129, 1025, 9000, 70001])
def test_tsqr_edges(m, k):
    g = torch.Generator(device="cuda").manual_seed(100 * m + k)
    A = torch.randn(k, m, generator=g, device="cuda").t()
    if k > 2:
        A[:, k // 2] = 0
        A[:, k - 1] = A[:, 0]
    R = ht.tsqr(A).double()
    assert torch.isfinite(R).all() and (torch.tril(R, -1) == 0).all() and (torch.diagonal(R) >= 0).all()
    G = A.double().t() @ A.double()
    d = torch.diagonal(G).sqrt().clamp_min(1e-30)
    assert (((R.t() @ R - G) / d[:, None] / d[None]).abs().max()) < 2.9e-5
