"""The exact-fp32 weight gradient at the edges of its chunks of 64 and 128 pairs, for widths of each of its three forms (by
the shared memory a chunk takes), on offsets of none to three chunks.  Whole numbers of at most 3 keep every sum below 2^24: exact."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu

COUNTS = [1, 63, 64, 65, 0, 127, 128, 129, 191, 192, 193, 255, 256, 257, 383, 384, 385]


@pytest.mark.parametrize("c_in,c_out", [(3, 5), (16, 16), (24, 24), (20, 36), (9, 64), (33, 40), (64, 64), (65, 70)])
def test_sums_are_exact_at_the_edges_of_chunks(c_in, c_out):
    p = Problem(_map(500, COUNTS, 3), c_in, c_out, seed=1, mode="fp32")
    gen = torch.Generator(device="cuda").manual_seed(5)
    p.feats, p.grad_out = (torch.randint(-3, 4, t.shape, generator=gen, device="cuda").to(t.dtype) for t in (p.feats, p.grad_out))
    backend.device_status(reset=True)
    grad = torch.zeros((len(COUNTS), c_in, c_out), device="cuda")
    backend.fgms_wgrad_cuda(p.feats, p.grad_out, grad, p.kpos, p.imap, p.omap, False)
    at = 0
    for k, n in enumerate(COUNTS):
        i, o = p.imap[at:at + n].long(), p.omap[at:at + n].long()
        assert torch.equal(grad[k].double(), p.feats[i].double().T @ p.grad_out[o].double())
        at += n
    assert backend.device_status(reset=True) == 0
