"""The autograd function of ``nn.sparse_conv``: which gradients it computes, what it does with what autograd hands it, and
the module switch it follows."""
import threading

import numpy as np
import pytest
import torch

from fgms_b200 import backend, clouds, gpu_maps, maps, nn
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    coords = clouds.uniform_cloud(2500, 18, 21)
    return maps.build_submanifold_map(coords, 3), gpu_maps.build_submanifold_map(torch.from_numpy(coords).cuda(), 3)


@pytest.mark.parametrize("at_backward", [False, True])
def test_the_sums_of_a_backward_follow_the_switch_as_it_is_then(scene, at_backward):
    """``backend.WGRAD_FP32_SUMS`` decides at the backward pass, whatever it was at the forward pass: the form with
    fp32 sums has one kernel more (the final addition)."""
    hk, dk = scene
    p = Problem(hk, 32, 32, seed=4, mode="fp16")
    weight = p.weights.clone().requires_grad_(True)
    try:
        backend.WGRAD_FP32_SUMS = not at_backward
        out = nn.sparse_conv(p.feats, weight, dk)
        backend.WGRAD_FP32_SUMS = at_backward
        before = backend.launch_count()
        out.backward(p.grad_out)
        launches = backend.launch_count() - before
    finally:
        backend.WGRAD_FP32_SUMS = False
    assert launches == (3 if at_backward else 2)  # clear, weight gradient, final addition; the input needs no gradient
    assert err(weight.grad, p.ref_wgrad()) <= TOL["fp16"]


@pytest.mark.parametrize("mode", ["fp16", "tf32", "fp32"])
@pytest.mark.parametrize("of_input,of_weight", [(True, False), (False, True), (True, True)])
def test_only_the_gradients_that_are_asked_for(scene, mode, of_input, of_weight):
    hk, dk = scene
    p = Problem(hk, 32, 16, seed=4, mode=mode)
    feats, weight = p.feats.clone().requires_grad_(of_input), p.weights.clone().requires_grad_(of_weight)
    nn.sparse_conv(feats, weight, dk, arch80=p.arch80).backward(p.grad_out)
    assert (feats.grad is not None, weight.grad is not None) == (of_input, of_weight)
    assert not of_input or err(feats.grad, p.ref_dgrad()) <= TOL[mode]
    assert not of_weight or err(weight.grad, p.ref_wgrad()) <= TOL[mode]


def test_the_gradient_of_one_of_two_that_require_it(scene):
    hk, dk = scene
    p = Problem(hk, 32, 16, seed=4, mode="tf32")
    feats, weight = p.feats.clone().requires_grad_(), p.weights.clone().requires_grad_()
    out = nn.sparse_conv(feats, weight, dk)
    (got,) = torch.autograd.grad(out, (weight,), p.grad_out, retain_graph=True)
    assert err(got, p.ref_wgrad()) <= TOL["tf32"]
    (got,) = torch.autograd.grad(out, (feats,), p.grad_out)
    assert err(got, p.ref_dgrad()) <= TOL["tf32"]


def test_output_gradients_and_inputs_of_other_layouts(scene):
    """Columns-first and expanded output gradients, columns-first features and weights: the results of contiguous ones."""
    hk, dk = scene
    p = Problem(hk, 32, 16, seed=4, mode="tf32")
    columns_first = lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2)
    feats, weight = columns_first(p.feats).requires_grad_(), columns_first(p.weights).requires_grad_()
    out = nn.sparse_conv(feats, weight, dk)
    assert err(out, p.ref_fwd()) <= TOL["tf32"]
    out.backward(columns_first(p.grad_out), retain_graph=True)
    assert err(feats.grad, p.ref_dgrad()) <= TOL["tf32"] and err(weight.grad, p.ref_wgrad()) <= TOL["tf32"]
    feats.grad = weight.grad = None
    out.sum().backward()
    p.g_np = np.ones_like(p.g_np)
    assert err(feats.grad, p.ref_dgrad()) <= TOL["tf32"] and err(weight.grad, p.ref_wgrad()) <= TOL["tf32"]


def _train(p, dk, stream, reps, got):
    with torch.cuda.stream(stream):
        for _ in range(reps):
            feats, weight = p.feats.clone().requires_grad_(), p.weights.clone().requires_grad_()
            out = nn.sparse_conv(feats, weight, dk, arch80=p.arch80)
            got.append((out.detach(), *torch.autograd.grad(out, (feats, weight), p.grad_out)))


@pytest.mark.parametrize("mode", ["fp16", "fp32"])
def test_side_streams_and_two_threads(scene, mode):
    """Two threads, each with a stream and a layer width of its own: every pass gives its layer's results."""
    hk, dk = scene
    problems = [Problem(hk, 32, 16, seed=4, mode=mode), Problem(hk, 64, 48, seed=5, mode=mode)]
    got, streams = [[], []], [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=_train, args=(p, dk, s, 10, g)) for p, s, g in zip(problems, streams, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for p, passes in zip(problems, got):
        assert len(passes) == 10
        want = p.ref_fwd(), p.ref_dgrad(), p.ref_wgrad()
        for tensors in passes:
            assert all(err(a, b) <= TOL[mode] for a, b in zip(tensors, want))


@pytest.mark.parametrize("a_bytes", [0, 1, 15, 16, 17, 4096, 70001])
@pytest.mark.parametrize("b_bytes", [0, 2, 16, 31, 5000])
def test_two_buffers_of_any_size_are_cleared_and_nothing_else(a_bytes, b_bytes):
    from fgms_b200 import _lib
    a, b = (torch.full((n + 64,), 7, dtype=torch.uint8, device="cuda") for n in (a_bytes, b_bytes))
    _lib.check(_lib.lib.fgms_b200_zero2(a.data_ptr() if a_bytes else None, a_bytes, b.data_ptr() if b_bytes else None, b_bytes,
                                        torch.cuda.current_stream().cuda_stream))
    for t, n in ((a, a_bytes), (b, b_bytes)):
        assert int(t[:n].sum()) == 0 and bool((t[n:] == 7).all())
