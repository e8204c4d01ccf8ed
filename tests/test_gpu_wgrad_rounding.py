"""How often an fp16 weight gradient is rounded (short rows, ``csrc/rows_wgrad.cuh``): an offset of up to 256 pairs is
one fp16 addition.  Whole-number inputs make every fp32 sum exact (256 products of at most 900 stay below 2^24), so a
gradient that is rounded once equals the exact sum rounded to fp16, bit for bit; partial sums rounded on the way do not."""
import numpy as np
import pytest
import torch

from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu


def _whole_numbers(p, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for name in ("feats", "grad_out"):
        t = getattr(p, name)
        setattr(p, name, torch.randint(-30, 31, t.shape, generator=gen, device="cuda").to(t.dtype))


def _exact(p, k):
    a, b = int(p.km.kpos[k]), int(p.km.kpos[k + 1])
    return p.feats[p.imap[a:b].long()].double().T @ p.grad_out[p.omap[a:b].long()].double()


@pytest.mark.parametrize("counts", [[80] * 27, [256] * 27, [1, 255, 0, 17, 129, 240, 16, 256, 2], [40] * 125, [100000] + [80] * 26])
@pytest.mark.parametrize("c_in,c_out", [(32, 32), (16, 64), (48, 48), (64, 64)])
def test_an_offset_of_up_to_256_pairs_is_rounded_once(counts, c_in, c_out):
    p = Problem(_map(max(max(counts), 600), counts, 11), c_in, c_out, seed=3, mode="fp16")
    _whole_numbers(p, 7)
    _, w_grad = p.run_bwd()
    for k, n in enumerate(counts):
        if n <= 256:
            want = _exact(p, k)
            assert float(want.abs().max()) < 65504
            assert torch.equal(w_grad[k], want.half()), f"offset {k} of {n} pairs"


def test_tiles_side_by_side_are_rounded_no_more_often():
    """Rows beyond half of L2 (tiles handed out side by side), small offsets between large ones."""
    counts = [200, 60000, 0, 80, 120000, 256]
    n = (72 << 20) // (64 * 2)
    p = Problem(_map(n, counts, 5), 32, 32, seed=2, mode="fp16")
    _whole_numbers(p, 9)
    _, w_grad = p.run_bwd()
    for k, c in enumerate(counts):
        if c <= 256:
            assert torch.equal(w_grad[k], _exact(p, k).half()), f"offset {k} of {c} pairs"
