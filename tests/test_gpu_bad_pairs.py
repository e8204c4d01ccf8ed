"""Map entries no tensor has: every kernel skips the pair and counts it, also where both entries are -1 (the usual
"no neighbour" value) on the exact-fp32 kernels, as the CUDA-core kernels always did.  What a skipped pair names reaches
nothing, infinities and NaN included."""
import numpy as np
import pytest
import torch

from fgms_b200 import backend
from oracle import spconv_oracle as orc
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
    maps = (cut, p.km.imap[:keep], p.km.omap[:keep])
    backend.device_status(reset=True)
    out = p.run_fwd()
    assert backend.device_status() == 1
    in_grad, w_grad = p.run_bwd()
    assert backend.device_status() == 2  # once in each pass
    assert err(out, orc.fwd(p.f_np, p.w_np, p.km.n_out, *maps)) <= TOL["fp32"]
    assert err(in_grad, orc.dgrad(p.g_np, p.w_np, p.km.n_in, *maps)) <= TOL["fp32"]
    assert err(w_grad, orc.wgrad(p.f_np, p.g_np, p.km.k_vol, *maps)) <= TOL["fp32"]


@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 32, 48), ("tf32", 32, 16), ("fp32", 20, 36)])
def test_infinities_and_nans_stay_in_their_pairs(mode, c_in, c_out):
    """A row of NaN that only a skipped pair names reaches nothing; infinite and NaN rows of real pairs reach exactly the
    values they reach in the oracle."""
    p = Problem(_map(400, COUNTS, 3), c_in, c_out, seed=2, mode=mode)
    last = p.km.pairs - 1
    skipped_in, skipped_out = int(p.km.imap[last]), int(p.km.omap[last])
    for name, rows in (("imap", skipped_in), ("omap", skipped_out)):  # no other pair names these rows
        m = getattr(p.km, name)
        m[:last][m[:last] == rows] = (rows + 1) % 400
        getattr(p, name).copy_(torch.from_numpy(m))
    p.omap[last] = 400  # no such row
    for t, np_t, row in ((p.feats, p.f_np, skipped_in), (p.grad_out, p.g_np, skipped_out)):
        t[row] = float("nan")
        np_t[row] = 0  # the oracle does without the pair
        t[5, 3], np_t[5, 3] = float("inf"), np.inf
        t[9, 1], np_t[9, 1] = float("nan"), np.nan
    cut = p.km.kpos.copy()
    cut[-1] = last
    maps = (cut, p.km.imap[:last], p.km.omap[:last])
    with np.errstate(invalid="ignore"):
        want = (orc.fwd(p.f_np, p.w_np, p.km.n_out, *maps), orc.dgrad(p.g_np, p.w_np, p.km.n_in, *maps),
                orc.wgrad(p.f_np, p.g_np, p.km.k_vol, *maps))
    for got, ref in zip((p.run_fwd(), *p.run_bwd()), want):
        got = got.double().cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
        assert np.isfinite(ref).sum() > 0.5 * ref.size
