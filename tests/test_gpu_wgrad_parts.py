"""The tcgen05 weight gradient where several CTAs share an offset's gradient, each a block of its channels: pair counts on both sides
of the lines that decide it, on all SMs and on a backward's share of them.  Whole numbers of at most 3 keep every sum below 2^24,
so the fp32 sums have to be exact."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


def _problem(stages, mode, c_in, c_out):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = max(1, int(128 * stages * sms) - 7)
    p = Problem(_map(pairs + 2, [pairs // 3, pairs - pairs // 3], 3), c_in, c_out, seed=1, mode=mode)
    gen = torch.Generator(device="cuda").manual_seed(5)
    p.feats, p.grad_out = (torch.randint(-3, 4, t.shape, generator=gen, device="cuda").to(t.dtype) for t in (p.feats, p.grad_out))
    return p


@pytest.mark.parametrize("stages", [0, 0.3, 0.48, 0.6, 1.1, 1.3, 2.1, 2.4, 3.1, 3.4, 5.6])
@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 256, 256), ("fp16", 160, 192), ("fp16", 192, 64), ("fp16", 96, 224), ("fp16", 128, 96),
                                             ("fp16", 144, 256), ("tf32", 256, 160), ("tf32", 64, 256)])
def test_sums_are_exact_whatever_the_parts(stages, mode, c_in, c_out):
    p = _problem(stages, mode, c_in, c_out)
    pairs = p.imap.numel()
    backend.device_status(reset=True)
    p.omap[pairs // 2] = pairs + 2  # skipped, and counted once
    grad = torch.zeros((2, c_in, c_out), dtype=p.dtype, device="cuda")
    sums = backend.fgms_wgrad_cuda(p.feats, p.grad_out, grad, p.kpos, p.imap, p.omap, True, fp32_sums=True)
    got = sums[: 2 * c_in * c_out].view(2, c_in, c_out) if mode == "fp16" else grad
    keep = torch.arange(pairs, device="cuda") != pairs // 2
    at = [0] + p.kpos.tolist()[1:]
    for k in range(2):
        i, o, on = (t[at[k]:at[k + 1]] for t in (p.imap, p.omap, keep))
        assert torch.equal(got[k].double(), p.feats[i[on].long()].double().T @ p.grad_out[o[on].long()].double())
    assert backend.device_status(reset=True) == 1


@pytest.mark.parametrize("stages", [0.2, 1.2, 3.0])
@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 256, 256), ("fp16", 128, 256), ("tf32", 256, 128)])
def test_beside_the_input_gradient(stages, mode, c_in, c_out):
    p = _problem(stages, mode, c_in, c_out)
    in_grad, w_grad = p.run_bwd()
    p.f_np, p.g_np = p.feats.cpu().numpy(), p.grad_out.cpu().numpy()
    assert err(in_grad, p.ref_dgrad()) <= TOL[mode] and err(w_grad, p.ref_wgrad()) <= TOL[mode]
