"""The tcgen05 forward and input gradient where several CTAs share a tile's columns: pair counts on both sides of the line that
decides it, for two, three and four parts, one and two tiles a CTA, and entries outside the tensors counted once whatever the parts."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import _map
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tiles", [1, 2, lambda s: s // 4 - 1, lambda s: s // 4 + 1, lambda s: s // 2, lambda s: s // 2 + 2, lambda s: s, lambda s: 2 * s])
@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 128, 256), ("fp16", 256, 128), ("fp16", 192, 80), ("fp16", 96, 192), ("tf32", 64, 128), ("tf32", 128, 32)])
def test_parts_of_a_tile(mode, c_in, c_out, tiles):
    n = tiles if isinstance(tiles, int) else tiles(_sms())
    pairs = 128 * n - 5
    p = Problem(_map(pairs + 3, [pairs], 3), c_in, c_out, seed=n, mode=mode)
    backend.device_status(reset=True)
    assert err(p.run_fwd(), p.ref_fwd()) <= TOL[mode]
    in_grad, w_grad = p.run_bwd()
    assert err(in_grad, p.ref_dgrad()) <= TOL[mode] and err(w_grad, p.ref_wgrad()) <= TOL[mode]
    assert backend.device_status() == 0


def test_a_skipped_pair_is_counted_once():
    p = Problem(_map(700, [300, 200], 3), 256, 256, seed=2, mode="fp16")
    p.imap[17] = 700
    p.omap[301] = -3
    backend.device_status(reset=True)
    p.run_fwd()
    assert backend.device_status(reset=True) == 2


@pytest.mark.parametrize("rows", [1, 127, 129, lambda s: 128 * (s // 4 - 3) - 1, lambda s: 128 * (s // 2 - 2) + 1])
@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 128, 256), ("fp16", 96, 192), ("tf32", 64, 128)])
def test_parts_of_a_tile_with_a_separate_centre(mode, c_in, c_out, rows):
    """The centre's rows are a segment of their own, which the line counts too."""
    n = rows if isinstance(rows, int) else rows(_sms())
    p = Problem(_map(n, [min(n, c) for c in (40, 1, 0, 130, 7)], 3), c_in, c_out, seed=n, mode=mode)
    backend.device_status(reset=True)
    assert err(p.run_fwd(separate_mid=True, fused=False), p.ref_fwd(precompute=True)) <= TOL[mode]
    assert backend.device_status() == 0
