"""Map entries no tensor has: every kernel skips the pair and counts it, also where both entries are -1 (the usual
"no neighbour" value) on the exact-fp32 kernels, as the CUDA-core kernels always did."""
import pytest

from fgms_b200 import backend
from tests.test_gpu_rows import COUNTS, _map
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c_in,c_out", [(20, 36), (16, 16), (65, 130)])
def test_a_pair_of_minus_ones_is_counted_in_every_exact_fp32_pass(c_in, c_out):
    p = Problem(_map(400, COUNTS, 3), c_in, c_out, seed=2, mode="fp32")
    keep = p.km.pairs - 1  # the last pair of the last offset
    p.imap[keep] = p.omap[keep] = -1
    cut = p.km.kpos.copy()
    cut[-1] = keep
    from oracle import spconv_oracle as orc
    maps = (cut, p.km.imap[:keep], p.km.omap[:keep])
    backend.device_status(reset=True)
    out = p.run_fwd()
    assert backend.device_status() == 1
    in_grad, w_grad = p.run_bwd()
    assert backend.device_status() == 2  # once in each pass
    assert err(out, orc.fwd(p.f_np, p.w_np, p.km.n_out, *maps)) <= TOL["fp32"]
    assert err(in_grad, orc.dgrad(p.g_np, p.w_np, p.km.n_in, *maps)) <= TOL["fp32"]
    assert err(w_grad, orc.wgrad(p.f_np, p.g_np, p.km.k_vol, *maps)) <= TOL["fp32"]
