"""``fgms_b200_bwd`` runs its two passes side by side: both gradients of every family of kernels, with inputs written by the
kernel just ahead and results read by the one just behind, buffers that overlap (one pass behind the other, the input gradient
first), and a graph.  Whole numbers of at most 1 and few pairs a row keep every result exact."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu
SHAPES = [("fp16", 64, 64), ("fp16", 32, 16), ("fp16", 128, 128), ("fp16", 64, 96), ("fp16", 256, 256), ("tf32", 32, 64), ("tf32", 128, 64),
          ("tf32", 48, 64), ("fp32", 20, 36), ("fp32", 16, 16), ("fp16", 20, 24)]


def _problem(mode, c_in, c_out, counts):
    p = Problem(_map(max(counts), counts, 3), c_in, c_out, seed=1, mode=mode)
    gen = torch.Generator(device="cuda").manual_seed(9)
    draw = lambda t: torch.randint(-1, 2, t.shape, generator=gen, device="cuda").to(t.dtype)
    p.weights = draw(p.weights)
    return p, draw


def _want(p):
    f, g, w = p.feats.double(), p.grad_out.double(), p.weights.double()
    dx, dw, kpos = torch.zeros_like(f), torch.zeros_like(w), p.kpos.tolist()
    for k in range(w.size(0)):
        i, o = p.imap[kpos[k]: kpos[k + 1]].long(), p.omap[kpos[k]: kpos[k + 1]].long()
        dx.index_add_(0, i, g[o] @ w[k].T)
        dw[k] = f[i].T @ g[o]
    return dx, dw


def _bwd(p, dx, dw):
    backend.fgms_bwd_cuda(p.grad_out, p.feats, p.weights, p.qsum, dx, dw, p.kpos, p.qkpos, p.imap, p.omap, False, p.arch80)


@pytest.mark.parametrize("counts", [[1800, 0, 1500], [300, 1, 40, 2000, 2000]])
@pytest.mark.parametrize("mode,c_in,c_out", SHAPES)
def test_both_gradients_between_kernels_of_others(mode, c_in, c_out, counts):
    p, draw = _problem(mode, c_in, c_out, counts)
    dx, dw = torch.empty_like(p.feats), torch.empty_like(p.weights)
    for _ in range(4):
        feats, grad, big = draw(p.feats), draw(p.grad_out), torch.zeros(1 << 24, device="cuda")
        big.add_(1)  # keeps the stream busy while the next ones are enqueued
        p.feats.copy_(feats); p.grad_out.copy_(grad); dx.zero_(); dw.zero_()
        _bwd(p, dx, dw)
        got = dx + 0, dw + 0
        want = _want(p)
        assert torch.equal(got[0].double(), want[0]) and torch.equal(got[1].double(), want[1])


@pytest.mark.parametrize("mode,c_in,c_out", SHAPES)
def test_weights_written_by_the_kernel_just_ahead(mode, c_in, c_out):
    """What the input gradient reads without waiting for the weight gradient: weights (by TMA in the wide layers), map, gradient."""
    p, draw = _problem(mode, c_in, c_out, [1800, 0, 1500])
    p.feats = draw(p.feats)
    dx, dw = torch.zeros_like(p.feats), torch.zeros_like(p.weights)
    for _ in range(6):
        weights, grad, big = draw(p.weights), draw(p.grad_out), torch.zeros(1 << 24, device="cuda")
        turn = torch.randperm(1500, device="cuda").int()
        imap, omap = p.imap.clone(), p.omap.clone()
        imap[1800:], omap[1800:] = imap[1800:][turn.long()], omap[1800:][turn.long()]
        dx.zero_(); dw.zero_()
        big.add_(1)
        p.grad_out.copy_(grad); p.imap.copy_(imap); p.omap.copy_(omap); p.weights.copy_(weights)
        _bwd(p, dx, dw)
        got = dx + 0, dw + 0
        want = _want(p)
        assert torch.equal(got[0].double(), want[0]) and torch.equal(got[1].double(), want[1])


@pytest.mark.parametrize("mode,c,pairs", [("fp16", 64, 400_000), ("fp16", 128, 200_000), ("tf32", 64, 100_000)])
def test_shares_of_large_layers(mode, c, pairs):
    p, draw = _problem(mode, c, c, [pairs // 4] * 4)
    gen = torch.Generator(device="cuda").manual_seed(3)
    keep = torch.rand(p.grad_out.shape, generator=gen, device="cuda") < 0.02  # sums of a weight gradient below 2048
    p.feats, p.grad_out = draw(p.feats), draw(p.grad_out) * keep
    dx, dw = torch.zeros_like(p.feats), torch.zeros_like(p.weights)
    _bwd(p, dx, dw)
    want = _want(p)
    assert float(want[1].abs().max()) < 2048
    assert torch.equal(dx.double(), want[0]) and torch.equal(dw.double(), want[1])


def test_an_input_gradient_over_the_features_goes_first():
    p, draw = _problem("fp16", 64, 64, [1800, 1500])
    p.feats, p.grad_out = draw(p.feats), draw(p.grad_out)
    start = p.feats.clone()
    dx = torch.zeros_like(start)
    _bwd(p, dx, torch.zeros_like(p.weights))
    dw, want = torch.zeros_like(p.weights), torch.zeros_like(p.weights)
    _bwd(p, p.feats, dw)  # adds the input gradient to the features, then the weight gradient of the sum
    assert torch.equal(p.feats, start + dx)
    backend.fgms_wgrad_cuda(start + dx, p.grad_out, want, p.kpos, p.imap, p.omap, True)
    assert torch.allclose(dw.float(), want.float(), rtol=2e-3, atol=2.0)  # up to 1800 products of at most 65, rounded to 11 bits


def test_replayed_from_a_graph():
    p, draw = _problem("fp16", 128, 64, [1500, 900])
    dx, dw, after = torch.zeros_like(p.feats), torch.zeros_like(p.weights), torch.empty_like(p.feats)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _bwd(p, dx, dw)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            dx.zero_(); dw.zero_()
            _bwd(p, dx, dw)
            after.copy_(dx)
    for _ in range(3):
        p.feats.copy_(draw(p.feats)); p.grad_out.copy_(draw(p.grad_out))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = _want(p)
        assert torch.equal(after.double(), want[0]) and torch.equal(dw.double(), want[1])
