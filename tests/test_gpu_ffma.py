"""The exact-fp32 kernels (``csrc/ffma_rows.cuh``) where they can go wrong: widths that fill no unit of four or eight
channels, one channel, the widest they take and the next one (which the general kernel takes), blocks of 64 output
channels, offsets of 0 .. 300 pairs, the centre as a dense segment, rows that start off a 16-byte boundary."""
import pytest
import torch

from fgms_b200 import backend
from tests.test_gpu_rows import COUNTS, _map
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


def _check(p):
    # sums of at most 27 x 128 (forward, dgrad) or 300 (weight gradient) fp32 products
    backend.device_status(reset=True)
    assert err(p.run_fwd(), p.ref_fwd()) <= TOL["fp32"]
    in_grad, w_grad = p.run_bwd()
    assert err(in_grad, p.ref_dgrad()) <= TOL["fp32"] and err(w_grad, p.ref_wgrad()) <= TOL["fp32"]
    assert backend.device_status() == 0


@pytest.mark.parametrize("c_in,c_out", [(1, 1), (1, 130), (3, 16), (4, 33), (16, 16), (17, 3), (20, 36), (33, 2), (63, 65), (64, 64),
                                        (65, 9), (128, 128), (129, 12), (12, 129)])
def test_widths_at_tile_edges(c_in, c_out):
    _check(Problem(_map(400, COUNTS, 3), c_in, c_out, seed=c_in + c_out, mode="fp32"))


@pytest.mark.parametrize("counts", [[1], [0, 0, 5], [30000] * 4, [40] * 125])
@pytest.mark.parametrize("c_in,c_out", [(20, 36), (3, 24), (64, 4)])
def test_few_and_many_pairs(counts, c_in, c_out):
    _check(Problem(_map(31000, counts, 5), c_in, c_out, seed=9, mode="fp32"))


def test_dense_centre():
    p = Problem(_map(333, [50, 0, 60], 4), 20, 36, seed=1, mode="fp32")
    assert err(p.run_fwd(separate_mid=True), p.ref_fwd(precompute=True)) <= TOL["fp32"]


def test_rows_off_a_16_byte_boundary():
    p = Problem(_map(400, COUNTS, 3), 20, 36, seed=5, mode="fp32")
    want = p.run_fwd(), *p.run_bwd()
    for name in ("feats", "weights", "grad_out"):
        t = getattr(p, name)
        room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
        setattr(p, name, room[1:].view(t.shape).copy_(t))
    got = p.run_fwd(), *p.run_bwd()
    for a, b in zip(got, want):
        assert err(a, b.cpu().double().numpy()) <= TOL["fp32"]
