"""A layer call recorded in a CUDA graph: a replay on a batch with an infinity must
not leave the later replays on the path such batches take.  Values, and the time
of a replay (the path's products run several times slower)."""
import pytest
import torch

from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backward", [False, True])
def test_replay_after_a_batch_with_an_infinity(backward):
    g = torch.Generator(device="cuda").manual_seed(3)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n, m, r, batch = (8, 8, 16), (8, 8, 16), 16, 8192
    f = [rn(n[j], m[j], r) / 4 for j in range(3)] + [rn(r, r, r) / r, rn(r, r) / 4]
    x, dy = rn(batch, 1024), rn(batch, 1024)
    call = (lambda: htlayer.layer_backward(x, dy, *f)[0]) if backward else (lambda: htlayer.layer_forward(x, *f))
    for _ in range(2):   # the workspace is made outside the capture
        want = call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()

    def us():
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    clean = us()
    assert torch.equal(out, want)
    v = (dy if backward else x)
    keep = v[3, 5].clone()
    v[3, 5] = float("inf")
    graph.replay()
    torch.cuda.synchronize()
    assert not torch.isfinite(out[3]).any() and torch.isfinite(out[4:]).all()
    v[3, 5] = keep
    assert us() < 1.5 * clean
    assert torch.equal(out, want)
