"""Products of operands that have no BF16 planes (infinities, NaN, entries that
round up past the largest BF16): formed from the FP32 operands inside the same
launch (csrc/tc3_gemm.cu, t3_fallback), for every operand layout, output form and
tile width, forwards and backwards.

A layer of ranks 1 with n = (1, 1, N), m = (1, 1, M) has any N x M matrix as its
weight, and du3 of it is the weight's gradient.

Tolerance: FP32 chains of at most K terms, K 2^-24 of the terms' magnitudes.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def dense(w):
    one = torch.ones(1, 1, 1, device="cuda")
    return one, one, w.t().contiguous().unsqueeze(2), one, one[0]


def same(got, a, b):
    """got against a @ b (64 bits): the same infinities and NaN, finite entries to
    FP32 rounding of the sum's terms."""
    want = a.double() @ b.double()
    got = got.double()
    over = want.abs() > 3.4028235e38
    want[over] = want[over].sign() * INF
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[over].sign(), want[over].sign())
    fin = torch.isfinite(want)
    size = torch.where(torch.isfinite(a), a, 0).double().abs() @ torch.where(torch.isfinite(b), b, 0).double().abs()
    assert ((got - want).abs()[fin] <= a.shape[1] * 2.0 ** -24 * size[fin]).all()


# tiles of 64, 128 and 256 columns with remainders, K blocks of 64 with
# remainders, long K in several splits (the weight's gradient over 9000 rows)
@pytest.mark.parametrize("N,M,batch", [(8, 8, 1), (64, 96, 70), (72, 120, 129), (104, 112, 700), (1024, 8, 65),
                                       (8, 1024, 300), (64, 64, 9000), (64, 192, 40000)])
@pytest.mark.parametrize("value", [INF, NAN, 3.4e38])
def test_layer(N, M, batch, value):
    g = torch.Generator(device="cuda").manual_seed(N + M + batch)
    x, w, dy = randn(g, batch, N), randn(g, M, N), randn(g, batch, M)
    bias = randn(g, M)
    x[batch // 2, N // 3] = value
    f = dense(w)
    same(htlayer.layer_forward(x, *f), x, w.t())
    y = htlayer.layer_forward(x, *f, bias=bias, relu=True)
    z = htlayer.layer_forward(x, *f) + bias
    assert torch.equal(y, torch.fmax(z, torch.zeros_like(z)))
    dx, _, _, du3 = htlayer.layer_backward(x, dy, *f)[:4]
    same(dx, dy, w)
    same(du3[:, :, 0], x.t(), dy)
    x[batch // 2, N // 3] = 1.0
    dy[batch // 3, M // 2] = -value
    dx, _, _, du3 = htlayer.layer_backward(x, dy, *f)[:4]
    same(dx, dy, w)
    same(du3[:, :, 0], x.t(), dy)


def test_layer_weight_without_planes():
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w, dy = randn(g, 200, 64), randn(g, 96, 64), randn(g, 200, 96)
    w[5, 60] = -INF
    same(htlayer.layer_forward(x, *dense(w)), x, w.t())
    same(htlayer.layer_backward(x, dy, *dense(w))[0], dy, w)


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


# (1.4e9 multiply-adds take planes)
@pytest.mark.parametrize("dims,r", [((301, 260, 397), 64), ((640, 321, 420), 17)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
@pytest.mark.parametrize("leaf", [0, 1, 2])
def test_reconstruct(dims, r, make, leaf):
    """An infinity in one factor: whole slices of the tensor are infinite or NaN, the
    rest is what it is without it."""
    g = torch.Generator(device="cuda").manual_seed(2)
    tr = make([1, r, r, r, r])
    U = {t: cm(randn(g, dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    B = {t: cm(randn(g, r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}
    clean = ht.reconstruct(tr, U, B, dims)
    t = tr.leaves()[leaf]
    U[t][7, 3] = INF
    X = ht.reconstruct(tr, U, B, dims)
    mode = 2 - tr.modes[t][0]
    hit = X.select(mode, 7)
    assert not torch.isfinite(hit).any()
    rest = torch.ones(X.shape[mode], dtype=torch.bool, device="cuda")
    rest[7] = False
    a, b = X.movedim(mode, 0)[rest].double(), clean.movedim(mode, 0)[rest].double()
    assert float((a - b).norm() / b.norm()) < 2e-6   # FP32 chains of at most 64 terms against planes, three products


@pytest.mark.parametrize("batch", [128, 8192])
def test_call_is_not_slow(batch):
    """A batch with an infinity in it takes a small multiple of a finite one (3 to 5: the
    CUDA cores' rate), not the hundreds of one output at a time from global memory."""
    g = torch.Generator(device="cuda").manual_seed(3)
    n, m, r = (8, 8, 16), (8, 8, 16), 16
    f = [randn(g, n[j], m[j], r) / 4 for j in range(3)] + [randn(g, r, r, r) / r, randn(g, r, r) / 4]
    x = randn(g, batch, 1024)

    def us():
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                htlayer.layer_forward(x, *f)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    clean = us()
    x[3, 5] = INF
    assert us() < 12 * clean
