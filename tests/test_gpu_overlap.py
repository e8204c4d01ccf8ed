"""What runs beside the short-row kernels: the exchange of the ranks' sums beside the backward it is meant to hide
behind, and kernels of other streams on the SMs ``fgms_b200_set_reserved_sms`` keeps free."""
import pytest
import torch

from fgms_b200 import _lib, backend
from fgms_b200.dist import PeerExchange

pytestmark = pytest.mark.gpu


class _Layer:
    """A layer whose passes take some hundred microseconds: 27 offsets of 300 k pairs each, of more where rows are short."""

    def __init__(self, c_in, c_out, dtype):
        n = max(400_000, 25_600_000 // (c_in + c_out))
        per = n * 3 // 4
        gen = torch.Generator(device="cuda").manual_seed(4)
        rows = lambda c: torch.randn((n, c), generator=gen, device="cuda").to(dtype)
        self.feats, self.grad_out, self.in_grad = rows(c_in), rows(c_out), torch.zeros((n, c_in), dtype=dtype, device="cuda")
        self.weight = torch.randn((27, c_in, c_out), generator=gen, device="cuda").to(dtype) * 0.05
        pick = lambda: torch.randperm(n, generator=gen, device="cuda")[:per].sort().values.int()
        self.imap = torch.cat([pick() for _ in range(27)])
        self.omap = torch.cat([pick() for _ in range(27)])
        self.kpos = torch.arange(28, device="cuda", dtype=torch.int32) * per

    def wgrad(self):
        backend.fgms_wgrad_cuda(self.feats, self.grad_out, torch.zeros_like(self.weight), self.kpos, self.imap, self.omap, True)

    def dgrad(self):
        backend.fgms_dgrad_cuda(self.grad_out, self.weight, self.in_grad, self.kpos, self.imap, self.omap, True)

    def bwd(self):
        backend.fgms_bwd_cuda(self.grad_out, self.feats, self.weight, 0, self.in_grad, torch.zeros_like(self.weight), self.kpos, None,
                              self.imap, self.omap, False, True)


def _side_and_main_ms(call, side, beside):
    """Times from the start of ``call()`` to the end of ``beside()`` on ``side`` and of the call itself."""
    main = torch.cuda.current_stream()
    start, end_side, end_main = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    torch.cuda.synchronize()
    start.record()
    side.wait_event(start)
    call()
    with torch.cuda.stream(side):
        # the call fills the chip before the other kernel is let go
        torch.cuda._sleep(60_000)
        beside()
        end_side.record(side)
    end_main.record(main)
    torch.cuda.synchronize()
    return start.elapsed_time(end_side), start.elapsed_time(end_main)


@pytest.mark.parametrize("pass_", ["dgrad", "wgrad"])
@pytest.mark.parametrize("c_in,c_out,dtype", [(32, 32, torch.float16), (64, 64, torch.float16), (16, 16, torch.float16),
                                              (32, 32, torch.float32), (48, 16, torch.float16), (64, 32, torch.float32)])
def test_the_exchange_runs_beside_the_backward(pass_, c_in, c_out, dtype):
    layer = _Layer(c_in, c_out, dtype)
    call = getattr(layer, pass_)
    side = torch.cuda.Stream(priority=-1)
    px = PeerExchange(27 * c_in * c_out, "cuda")
    px.run(side)
    call()
    best = min((_side_and_main_ms(call, side, lambda: px.run(side)) for _ in range(5)), key=lambda t: t[0] / t[1])
    assert best[0] < 0.85 * best[1], f"the exchange ended after {best[0]:.3f} ms, the {pass_} after {best[1]:.3f} ms"


@pytest.mark.parametrize("c_in,c_out", [(32, 32), (64, 64)])
def test_reserved_sms_are_free_for_another_stream(c_in, c_out):
    """A kernel whose blocks need most of an SM's registers (softmax over long rows: 1024 threads each) finds room."""
    layer = _Layer(c_in, c_out, torch.float16)
    side = torch.cuda.Stream(priority=-1)
    x = torch.randn((8, 16384), device="cuda")
    torch.softmax(x, 1)
    try:
        assert _lib.lib.fgms_b200_set_reserved_sms(16) == 0
        layer.dgrad()
        best = min((_side_and_main_ms(layer.dgrad, side, lambda: torch.softmax(x, 1)) for _ in range(5)), key=lambda t: t[0] / t[1])
    finally:
        _lib.lib.fgms_b200_set_reserved_sms(0)
    assert best[0] < 0.75 * best[1], f"the other kernel ended after {best[0]:.3f} ms, the input gradient after {best[1]:.3f} ms"


@pytest.mark.parametrize("c_in,c_out", [(32, 32), (64, 64), (128, 128)])
def test_reserved_sms_are_free_throughout_a_backward(c_in, c_out):
    """The same kernel beside both gradients of one call, let go while the first of them runs."""
    layer = _Layer(c_in, c_out, torch.float16)
    side = torch.cuda.Stream(priority=-1)
    x = torch.randn((8, 16384), device="cuda")
    torch.softmax(x, 1)
    try:
        assert _lib.lib.fgms_b200_set_reserved_sms(16) == 0
        layer.bwd()
        best = min((_side_and_main_ms(layer.bwd, side, lambda: torch.softmax(x, 1)) for _ in range(5)), key=lambda t: t[0] / t[1])
    finally:
        _lib.lib.fgms_b200_set_reserved_sms(0)
    assert best[0] < 0.4 * best[1], f"the other kernel ended after {best[0]:.3f} ms, the backward after {best[1]:.3f} ms"
