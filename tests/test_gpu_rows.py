"""The short-row kernels (``csrc/rows_gms.cuh``, ``csrc/rows_wgrad.cuh``) at the edges of their tiles: offsets of 0 .. 33
pairs around the tiles of 16 and 32, every width of 16 .. 64 channels, the centre as a dense segment, and tiles handed
out side by side (rows that exceed half of L2)."""
import numpy as np
import pytest
import torch

from fgms_b200 import maps
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu
COUNTS = [0, 1, 15, 16, 17, 0, 31, 32, 33, 300, 2]


def _map(n, counts, seed):
    rng = np.random.default_rng(seed)
    pick = lambda c: np.sort(rng.choice(n, size=c, replace=False)).astype(np.int64)
    return maps._assemble(n, n, [(rng.permutation(pick(c)), pick(c)) for c in counts], None)


def _check(p):
    # bounds of the operator: sums of at most 64 products (forward, dgrad) or 300 (wgrad) per offset
    from fgms_b200 import backend
    backend.device_status(reset=True)
    unaligned = backend.fallback_count()
    tol = TOL["fp16" if p.dtype == torch.float16 else "tf32"]
    assert err(p.run_fwd(), p.ref_fwd()) <= tol
    in_grad, w_grad = p.run_bwd()
    assert err(in_grad, p.ref_dgrad()) <= tol and err(w_grad, p.ref_wgrad()) <= tol
    assert backend.device_status() == 0 and backend.fallback_count() == unaligned


@pytest.mark.parametrize("mode", ["fp16", "tf32"])
@pytest.mark.parametrize("c_in", [16, 32, 48, 64])
@pytest.mark.parametrize("c_out", [16, 32, 48, 64])
def test_every_width_at_tile_edges(mode, c_in, c_out):
    _check(Problem(_map(400, COUNTS, 3), c_in, c_out, seed=c_in + c_out, mode=mode))


@pytest.mark.parametrize("counts", [[1], [16], [0, 0, 5], [2000] * 3, [40] * 125])
def test_few_and_many_offsets(counts):
    _check(Problem(_map(2100, counts, 5), 32, 48, seed=9, mode="fp16"))


@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 64, 32), ("tf32", 32, 32)])
def test_tiles_side_by_side_when_rows_exceed_l2(mode, c_in, c_out):
    n = (72 << 20) // ((c_in + c_out) * (2 if mode == "fp16" else 4))
    _check(Problem(_map(n, [40, 3000, 0, 17, 60000, 1, 9000], 7), c_in, c_out, seed=2, mode=mode))


@pytest.mark.parametrize("counts", [[16384, 16383], [16384, 16384]])
def test_both_sides_of_the_line_of_tf32_32_to_64(counts):
    _check(Problem(_map(20000, counts, 3), 32, 64, seed=1, mode="tf32"))


def test_dense_centre():
    p = Problem(_map(333, [50, 0, 60], 4), 48, 32, seed=1, mode="fp16")
    assert err(p.run_fwd(separate_mid=True), p.ref_fwd(precompute=True)) <= TOL["fp16"]


@pytest.mark.parametrize("separate_mid", [False, True])
def test_many_tiles_a_warp_side_by_side(separate_mid):
    """Shares of a dozen tiles and more over offsets of very different lengths, with the centre as a dense segment too."""
    n = (72 << 20) // (64 * 2)
    p = Problem(_map(n, [300000, 0, 300000, 5, 300000, 70, 300000], 7), 32, 32, seed=2, mode="fp16")
    if separate_mid:
        assert err(p.run_fwd(separate_mid=True), p.ref_fwd(precompute=True)) <= TOL["fp16"]
    else:
        _check(p)
