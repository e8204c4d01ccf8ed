"""The output-stationary forward where its walk changes shape: rings of fewer stages than producer warps, rows of several and
of partly filled 128-byte chunks, several groups of tiles in a CTA, tiles of one row, offsets without any neighbour, and
rows without a neighbour beside rows that hold infinities."""
import numpy as np
import pytest
import torch

from fgms_b200 import maps
from tests.util import TOL, Problem, err

pytestmark = pytest.mark.gpu


def _map(n, seed):
    """Four offsets: every row, a third of the rows, none, one row."""
    rng = np.random.default_rng(seed)
    o = [np.arange(n), np.sort(rng.choice(n, max(1, n // 3), replace=False)), np.zeros(0, np.int64), np.array([n - 1])]
    i = [rng.permutation(n), rng.integers(0, n, o[1].size), np.zeros(0, np.int64), np.array([0])]
    knnz = np.array([x.size for x in o], np.int32)
    return maps.KernelMap(n, n, 4, knnz, np.concatenate([[0], np.cumsum(knnz)]).astype(np.int32), np.concatenate(i).astype(np.int32),
                          np.concatenate(o).astype(np.int32))


def _run(p, accumulate=False, start=7.0):
    from fgms_b200 import backend
    nbr = backend.build_neighbor_table(p.kpos, p.imap, p.omap, p.km.n_in, p.km.n_out)
    out = torch.full((p.km.n_out, p.c_out), start, dtype=p.dtype, device="cuda")
    backend.device_status(reset=True)
    backend.fgms_fwd_os_cuda(p.feats, p.weights, out, nbr, p.arch80, accumulate=accumulate)
    assert backend.device_status() == 0
    return out


# (256, 256): four stages and one weight buffer in fp16; (128, 128): nine; (64, 32): twelve, eight tiles to a group
@pytest.mark.parametrize("mode,c_in,c_out", [("fp16", 256, 256), ("fp16", 128, 128), ("fp16", 64, 32), ("fp16", 80, 48),
                                             ("tf32", 128, 128), ("tf32", 256, 32), ("tf32", 48, 16)])
@pytest.mark.parametrize("n", [1, 129, 40000])
def test_parity(mode, c_in, c_out, n):
    p = Problem(_map(n, n + c_in), c_in, c_out, seed=c_in + c_out, mode=mode)
    assert err(_run(p), p.ref_fwd()) <= TOL[mode]


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def test_many_groups_of_tiles():
    n = _sms() * 128 * 9 + 77  # nine and ten tiles of 32 channels in a CTA: two groups
    p = Problem(_map(n, 3), 16, 32, seed=5, mode="fp16")
    assert err(_run(p), p.ref_fwd()) <= TOL["fp16"]


@pytest.mark.parametrize("accumulate", [False, True])
def test_a_single_tile_behind_a_full_group(accumulate):
    n = _sms() * 128 * 9 - 40  # nine tiles in every CTA: eight at a time, then one, a single stage per offset
    p = Problem(_map(n, 4), 64, 32, seed=6, mode="fp16")
    start = 0.25 if accumulate else 0.0
    out = _run(p, accumulate=accumulate, start=0.25 if accumulate else 7.0)
    assert err(out, p.ref_fwd() + start) <= TOL["fp16"]


def test_rows_without_a_neighbour_see_nothing_of_the_others():
    p = Problem(_map(700, 9), 64, 64, seed=2, mode="fp16")
    clean = _run(p)
    last = int(p.km.imap[699])  # the input row of output row 699 under offset 0
    p.feats[last] = float("inf")
    out = _run(p)
    touched = np.unique(p.km.omap[p.km.imap == last])
    rest = np.setdiff1d(np.arange(700), touched)
    assert torch.equal(out[rest], clean[rest])
    assert (~torch.isfinite(out[touched])).any(dim=1).all()  # every row that has the pair
