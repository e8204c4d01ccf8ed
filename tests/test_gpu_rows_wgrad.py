"""The ring of tiles of the short-row weight gradient (``csrc/rows_wgrad.cuh``): shares of fewer tiles than a ring
holds, of as many, of one more, and of several rounds, a last tile of one pair, and entries outside the tensors on the way.
Whole numbers of at most 3 keep every sum below 2^24, so the fp32 sums have to be exact."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_per_warp", [0, 1, 2, 3, 4, 5, 7, 8, 9])
@pytest.mark.parametrize("mode,c_in,c_out,warps", [("fp16", 16, 16, 16), ("fp16", 32, 32, 16), ("fp16", 48, 32, 16), ("fp16", 48, 48, 12),
                                                   ("fp16", 64, 64, 8), ("tf32", 16, 16, 16), ("tf32", 32, 32, 16), ("tf32", 48, 48, 12),
                                                   ("tf32", 32, 64, 12), ("tf32", 48, 16, 16)])
def test_sums_are_exact_whatever_the_ring_holds(tiles_per_warp, mode, c_in, c_out, warps):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = 16 * sms * (warps * tiles_per_warp + 1) + 1
    p = Problem(_map(pairs, [pairs], 3), c_in, c_out, seed=1, mode=mode)
    gen = torch.Generator(device="cuda").manual_seed(5)
    p.feats, p.grad_out = (torch.randint(-3, 4, t.shape, generator=gen, device="cuda").to(t.dtype) for t in (p.feats, p.grad_out))
    backend.device_status(reset=True)
    imap = p.imap.clone()
    skipped = torch.arange(7, pairs, 1013, device="cuda")
    imap[skipped] = pairs
    grad = torch.zeros((1, c_in, c_out), dtype=p.dtype, device="cuda")
    sums = backend.fgms_wgrad_cuda(p.feats, p.grad_out, grad, p.kpos, imap, p.omap, True, fp32_sums=True)
    keep = torch.ones(pairs, dtype=torch.bool, device="cuda")
    keep[skipped] = False
    want = p.feats[p.imap[keep].long()].double().T @ p.grad_out[p.omap[keep].long()].double()
    got = sums[: c_in * c_out].view(c_in, c_out) if mode == "fp16" else grad[0]
    assert torch.equal(got.double(), want)
    assert backend.device_status(reset=True) == skipped.numel()
