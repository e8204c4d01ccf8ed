"""Both gradients of short fp16 rows by one kernel (``csrc/rows_wgrad.cuh``) on the fewest pairs it takes and on a few more, in offsets
of none, one, and a part of a tile, with entries outside the tensors, and the calls beside it that keep two kernels.  Numbers of
-1, 0 and 1 keep the input gradient's fp16 sums below 2^11 and the weight gradient's fp32 sums exact: it is rounded once."""
import gc

import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import Problem

pytestmark = pytest.mark.gpu
ROWS = 1 << 17
LEAST = [ROWS] * 8  # 2^20 pairs
SHAPES = [(16, 16), (16, 32), (32, 16), (32, 32), (48, 16), (16, 64), (64, 16), (32, 48), (48, 32), (64, 32), (32, 64)]


def _problem(c_in, c_out, counts):
    p = Problem(_map(ROWS, counts, 3), c_in, c_out, seed=1, mode="fp16")
    gen = torch.Generator(device="cuda").manual_seed(9)
    p.feats, p.grad_out, p.weights = (torch.randint(-1, 2, t.shape, generator=gen, device="cuda").half() for t in (p.feats, p.grad_out, p.weights))
    return p


def _check(p, launches, skip=()):
    """Gradients added to what is there already, and `launches` kernels for them."""
    imap, omap, keep = p.imap.clone(), p.omap.clone(), torch.ones(p.imap.numel(), dtype=torch.bool, device="cuda")
    for n, at in enumerate(skip):
        (imap, omap)[n % 2][at] = ROWS + n if n % 3 else -5
        keep[at] = False
    dx, dw = torch.ones_like(p.feats), torch.ones_like(p.weights)
    backend.device_status(reset=True)
    before = backend.launch_count()
    backend.fgms_bwd_cuda(p.grad_out, p.feats, p.weights, p.qsum, dx, dw, p.kpos, p.qkpos, imap, omap, False, p.arch80)
    assert backend.launch_count() - before == launches
    f, g, w, kpos = p.feats.double(), p.grad_out.double(), p.weights.double(), p.kpos.tolist()
    want_x, want_w = torch.ones_like(f), torch.ones_like(w)
    for k in range(w.size(0)):
        of = torch.arange(kpos[k], kpos[k + 1], device="cuda")[keep[kpos[k]: kpos[k + 1]]]
        i, o = imap[of].long(), omap[of].long()
        want_x.index_add_(0, i, g[o] @ w[k].T)
        want_w[k] += f[i].T @ g[o]
    assert torch.equal(dx.double(), want_x)
    if launches == 3:  # the clearing and the rounding of the sums beside it
        assert torch.equal(dw, want_w.half())
    else:  # a few roundings of at most 2^-11 of the largest sum each
        assert (dw.double() - want_w).abs().max() <= 8 * 2.0 ** -11 * max(want_w.abs().max(), 1)
    assert backend.device_status(reset=True) == 2 * len(skip)  # once in each gradient


@pytest.mark.parametrize("counts", [LEAST, LEAST + [0, 1, 0, 15, 16, 17, 300, 256, 257]])
@pytest.mark.parametrize("c_in,c_out", SHAPES)
def test_one_kernel_for_both(c_in, c_out, counts):
    _check(_problem(c_in, c_out, counts), 3, range(7, sum(counts), 200003))


@pytest.mark.parametrize("shape,counts", [((32, 32), [ROWS] * 7 + [ROWS - 1]), ((48, 48), LEAST), ((64, 48), LEAST)])
def test_fewer_pairs_and_longer_rows_keep_two_kernels(shape, counts):
    _check(_problem(*shape, counts), 2)


def test_weights_off_their_alignment_keep_two_kernels():
    p = _problem(32, 32, LEAST)
    shifted = torch.zeros(p.weights.numel() + 8, dtype=torch.float16, device="cuda")[1: 1 + p.weights.numel()].view_as(p.weights)
    p.weights = shifted.copy_(p.weights)
    _check(p, 2)


def test_without_memory_for_the_sums_two_kernels_run():
    p = _problem(32, 32, LEAST)
    dx, dw = torch.zeros_like(p.feats), torch.zeros_like(p.weights)
    gc.collect()  # what earlier tests left in cycles would otherwise be handed back at any time
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:  # nothing beyond what is reserved, and of that nothing that the 32 KB of the sums fit in
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)
        with pytest.raises(torch.OutOfMemoryError):
            while True:
                held.append(torch.empty(1 << 15, dtype=torch.uint8, device="cuda"))
        before = backend.launch_count()
        backend.fgms_bwd_cuda(p.grad_out, p.feats, p.weights, p.qsum, dx, dw, p.kpos, p.qkpos, p.imap, p.omap, False, p.arch80)
    finally:
        held.clear()
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert backend.launch_count() - before == 2
    want = torch.zeros_like(p.feats)
    backend.fgms_dgrad_cuda(p.grad_out, p.weights, want, p.kpos, p.imap, p.omap, p.arch80)
    assert torch.equal(dx, want) and float(dw.abs().max()) > 0
