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
