"""The pipelines of the output-stationary forward (``csrc/umma_osfwd.cuh``): CTAs of one tile and up (offsets dealt out to the
pipelines, then tiles), groups whose last one has fewer tiles than there are pipelines, fewer offsets than pipelines.  Values of -1, 0
and 1 keep every sum below 2048, so fp16 results have to be exact."""
import pytest
import torch

from fgms_b200 import backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c_in,c_out", [(64, 64), (128, 128), (32, 16), (48, 256)])
@pytest.mark.parametrize("k_vol", [1, 2, 3, 10])
@pytest.mark.parametrize("tiles", [0.3, 1, 1.5, 2, 3, 4.6, 7])
def test_exact_for_any_number_of_tiles_and_offsets(tiles, k_vol, c_in, c_out):
    _exact(tiles, k_vol, c_in, c_out, torch.half)


@pytest.mark.parametrize("dtype,c_in,c_out", [(torch.half, 144, 144), (torch.half, 160, 48), (torch.half, 208, 64), (torch.half, 256, 128),
                                              (torch.half, 224, 112), (torch.float, 32, 32), (torch.float, 64, 64), (torch.float, 80, 80),
                                              (torch.float, 208, 48), (torch.float, 160, 96)])
@pytest.mark.parametrize("k_vol", [3, 8])
@pytest.mark.parametrize("tiles", [0.3, 1.5, 3, 4.6])
def test_exact_for_wide_rows_and_tf32(tiles, k_vol, dtype, c_in, c_out):
    """Rows of up to seven 128-byte chunks, weights that leave rings of two slots and more; tf32 values as exact as fp16 ones."""
    _exact(tiles, k_vol, c_in, c_out, dtype)


def _exact(tiles, k_vol, c_in, c_out, dtype):
    n = int(torch.cuda.get_device_properties(0).multi_processor_count * 128 * tiles) - 5
    gen = torch.Generator(device="cuda").manual_seed(n + k_vol)
    draw = lambda *shape: torch.randint(-1, 2, shape, generator=gen, device="cuda").to(dtype)
    feats, weight, bias = draw(n, c_in), draw(k_vol, c_in, c_out), draw(c_out)
    nbr = torch.randint(-n // 2, n, (k_vol, (n + 127) // 128 * 128), generator=gen, device="cuda", dtype=torch.int32).clamp(min=-1)
    nbr[:, n:] = -1
    out = torch.full((n, c_out), 7.0, dtype=dtype, device="cuda")
    backend.device_status(reset=True)
    backend.fgms_fwd_os_cuda(feats, weight, out, nbr, True, bias=bias, relu=True)
    padded = torch.cat([feats, torch.zeros_like(feats[:1])])
    want = sum(padded[nbr[k, :n].long()].float() @ weight[k].float() for k in range(k_vol)) + bias.float()
    assert torch.equal(out.float(), want.clamp(min=0)) and backend.device_status() == 0
