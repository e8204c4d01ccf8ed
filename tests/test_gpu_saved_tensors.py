"""``nn.sparse_conv`` under saved-tensor hooks: what a hook hands back is checked like any argument, and hooks that move
the tensors elsewhere and back leave the gradients as they are."""
import pytest
import torch

from fgms_b200 import clouds, gpu_maps, maps, nn
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


def _layer():
    coords = clouds.uniform_cloud(2500, 18, 21)
    dk = gpu_maps.build_submanifold_map(torch.from_numpy(coords).cuda(), 3)
    p = Problem(maps.build_submanifold_map(coords, 3), 32, 64, seed=4, mode="tf32")
    return p, dk, p.feats.clone().requires_grad_(True), p.weights.clone().requires_grad_(True)


CHANGES = {
    "half_the_bytes": lambda t: t.half() if t.is_floating_point() else t,
    "columns_first": lambda t: t.t().contiguous().t() if t.dim() == 2 else t,
    "fewer_channels": lambda t: t[:, :16].contiguous() if t.dim() == 2 else t,
    "on_the_host": lambda t: t.cpu(),
    "short_maps": lambda t: t[:-1].contiguous() if t.dim() == 1 and t.numel() > 28 else (t[:5].contiguous() if t.dim() == 1 else t),
}


@pytest.mark.parametrize("name", list(CHANGES))
def test_a_hook_that_hands_back_something_else_is_an_error(name):
    p, dk, feats, weight = _layer()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, CHANGES[name]):
        out = nn.sparse_conv(feats, weight, dk)
    with pytest.raises(ValueError):
        out.backward(p.grad_out)


def test_tensors_saved_on_the_host_give_the_same_gradients():
    p, dk, feats, weight = _layer()
    with torch.autograd.graph.save_on_cpu():
        out = nn.sparse_conv(feats, weight, dk)
    out.backward(p.grad_out)
    assert err(feats.grad, p.ref_dgrad()) <= TOL["tf32"] and err(weight.grad, p.ref_wgrad()) <= TOL["tf32"]
