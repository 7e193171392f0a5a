"""TSQR of at most 32 columns at scales whose squares leave FP32's range, for whole
matrices, single columns and row blocks: R's error relative to the columns' norms
is that of entries of order one.

Tolerance as in test_gpu_tsqr_edges.py: 32 * 15 * 2^-24 = 2.9e-5.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht

pytestmark = pytest.mark.gpu
TOL = 2.9e-5


def check(A):
    R = ht.tsqr(A).double()
    assert torch.isfinite(R).all() and (torch.tril(R, -1) == 0).all() and (torch.diagonal(R) >= 0).all()
    G = A.double().t() @ A.double()
    d = torch.diagonal(G).sqrt()
    assert (((R.t() @ R - G) / d[:, None] / d[None]).abs().max()) < TOL


@pytest.mark.parametrize("m,k", [(64, 4), (100, 4), (33, 16), (5000, 8), (5000, 17), (9000, 32), (70001, 20)])
@pytest.mark.parametrize("scale", [1e25, 1e-15, 1e-18, 5e-20, 1e-20, 8e-21, 3e-21, 1e-25, 1e-30])
def test_scaled_matrix(m, k, scale):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    check((torch.randn(k, m, generator=g, device="cuda") * scale).t())


@pytest.mark.parametrize("k", [7, 16, 32])
def test_scaled_columns_and_rows(k):
    g = torch.Generator(device="cuda").manual_seed(k)
    A = torch.randn(k, 3000, generator=g, device="cuda")
    scales = torch.tensor([1.0, 1e-20, 1e10, 1e-27, 1e-4], device="cuda")
    check((A * scales[torch.arange(k, device="cuda") % 5, None]).t())
    B = torch.randn(k, 3000, generator=g, device="cuda") * 1e-22
    B[:, 2500:] *= 1e3   # row blocks of two tiny scales
    check(B.t())


def test_not_a_number_is_seen():
    A = torch.full((4, 200), 1e-25, device="cuda")
    A[1, 77] = float("nan")
    assert torch.isnan(ht.tsqr(A.t())).any()
