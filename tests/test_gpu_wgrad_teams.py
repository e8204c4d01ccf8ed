"""The producer teams of the tcgen05 weight gradient (``csrc/umma_wgrad3.cuh``): every number of 128-byte pieces a row may have,
packed stages, one team and two, shares of one stage (of 32 pairs, or up to four times that), of as many as the ring has slots (three
to five), and of several rounds (48 of 32 pairs: sixteen stages of 128), offsets that end inside a share, and entries
outside the tensors.  Whole numbers of at most 3 keep every sum below 2^24, so fp32 sums have to be exact."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu
WIDTHS = [("fp16", 128, 128), ("fp16", 96, 160), ("fp16", 256, 256), ("fp16", 16, 208), ("tf32", 64, 64), ("tf32", 48, 64),
          ("tf32", 96, 32), ("tf32", 160, 192), ("tf32", 256, 224), ("tf32", 16, 128), ("tf32", 144, 240)]


@pytest.mark.parametrize("stages", [0, 1, 2, 3, 4, 5, 9, 48])
@pytest.mark.parametrize("mode,c_in,c_out", WIDTHS)
def test_sums_are_exact_whatever_a_share_holds(mode, c_in, c_out, stages):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = 32 * sms * stages + 37
    counts = [pairs, 0, 1, pairs // 3 + 1]
    p = Problem(_map(pairs + 1, counts, 3), c_in, c_out, seed=1, mode=mode)
    gen = torch.Generator(device="cuda").manual_seed(5)
    p.feats, p.grad_out = (torch.randint(-3, 4, t.shape, generator=gen, device="cuda").to(t.dtype) for t in (p.feats, p.grad_out))
    assert backend.kernel_family("wgrad", c_in, c_out, p.dtype, True, len(counts)) == "tcgen05"
    backend.device_status(reset=True)
    omap = p.omap.clone()
    skipped = torch.arange(5, omap.numel(), 1013, device="cuda")
    omap[skipped] = -7
    grad = torch.zeros((len(counts), c_in, c_out), dtype=p.dtype, device="cuda")
    sums = backend.fgms_wgrad_cuda(p.feats, p.grad_out, grad, p.kpos, p.imap, omap, True, fp32_sums=True)
    got = (sums if mode == "fp16" else grad).reshape(-1)[: grad.numel()].view_as(grad).double()
    keep = torch.ones(omap.numel(), dtype=torch.bool, device="cuda")
    keep[skipped] = False
    kpos = p.kpos.tolist()
    for k in range(len(counts)):
        here = keep[kpos[k]: kpos[k + 1]]
        i, o = p.imap[kpos[k]: kpos[k + 1]][here].long(), p.omap[kpos[k]: kpos[k + 1]][here].long()
        assert torch.equal(got[k], p.feats[i].double().T @ p.grad_out[o].double()), f"offset {k}"
    assert backend.device_status(reset=True) == skipped.numel()
