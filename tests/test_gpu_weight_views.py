"""Weights that begin inside an allocation, 16-byte aligned and no more: the tcgen05 kernels that load them by TMA take them as
they take an allocation's start."""
import pytest
import torch

from fgms_b200 import clouds, maps
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 128, 128), ("fp16", 48, 80), ("fp16", 96, 32), ("tf32", 128, 64), ("tf32", 48, 80), ("tf32", 16, 96)])
def test_a_view_off_the_start(mode, c_in, c_out):
    from fgms_b200 import backend
    km = maps.build_submanifold_map(clouds.uniform_cloud(900, 12, seed=c_in + c_out), 3)
    p = Problem(km, c_in, c_out, seed=7, mode=mode)
    off = 16 // p.weights.element_size()
    buffer = torch.full((p.weights.numel() + 2 * off,), float("nan"), dtype=p.dtype, device="cuda")  # what lies beside is not read
    view = buffer[off:off + p.weights.numel()].view(p.weights.shape)
    view.copy_(p.weights)
    assert view.data_ptr() % 32 == 16
    p.weights = view
    left = backend.fallback_count()
    backend.device_status(reset=True)
    assert err(p.run_fwd(), p.ref_fwd()) <= TOL[mode]
    in_grad, w_grad = p.run_bwd()
    assert err(in_grad, p.ref_dgrad()) <= TOL[mode] and err(w_grad, p.ref_wgrad()) <= TOL[mode]
    out = torch.empty((km.n_out, c_out), dtype=p.dtype, device="cuda")
    backend.fgms_fwd_os_cuda(p.feats, view, out, backend.build_neighbor_table(p.kpos, p.imap, p.omap, km.n_in, km.n_out), p.arch80)
    assert err(out, p.ref_fwd()) <= TOL[mode]
    assert backend.fallback_count() == left and backend.device_status() == 0
