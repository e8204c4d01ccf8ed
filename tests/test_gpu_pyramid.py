"""The pyramid builder (``csrc/map_pyramid.cuh``): every map of every level equals the host builders' bit for bit, for rows
in any order, boxes around the 32-cell words of its bitmaps, and clouds it has to leave to the hash-table builders."""
import ctypes

import numpy as np
import pytest
import torch

from fgms_b200 import _lib, clouds, unet
from tests.test_gpu_maps import _dev, _same

pytestmark = pytest.mark.gpu


def _block(x, y, z):
    g = np.stack(np.meshgrid(np.arange(x), np.arange(y), np.arange(z), indexing="ij"), -1).reshape(-1, 3)
    return g.astype(np.int32)


CLOUDS = {
    "surface": lambda: clouds.surface_cloud(20000, 128, 5),
    "lidar": lambda: clouds.lidar_cloud(6, sweeps=1),
    "one": lambda: np.array([[-7, 0, 12]], dtype=np.int32),
    "column": lambda: _block(1, 1, 300) - np.array([5, 1, 33], dtype=np.int32),
    "z29": lambda: _block(3, 4, 29), "z30": lambda: _block(3, 4, 30), "z31": lambda: _block(3, 4, 31) + 31, "z62": lambda: _block(2, 9, 62) - 1,
    "far_apart": lambda: np.array([[0, 0, 0], [3, 900, 5], [700, 2, 1100]], dtype=np.int32),
    "too_large_a_box": lambda: np.concatenate([clouds.uniform_cloud(500, 20, 1), clouds.uniform_cloud(500, 20, 2) + 60000]).astype(np.int32),
}


def _check(dev_maps, host_maps):
    for d, h in zip(dev_maps.subm + dev_maps.down + dev_maps.up, host_maps.subm + host_maps.down + host_maps.up, strict=True):
        _same(d, h)
    for d, h in zip(dev_maps.down, host_maps.down):
        assert np.array_equal(d.out_coords.cpu().numpy(), h.out_coords)


@pytest.mark.parametrize("name", list(CLOUDS))
@pytest.mark.parametrize("levels", [1, 4])
def test_equals_the_host_builders(name, levels):
    coords = np.unique(CLOUDS[name](), axis=0)
    _check(unet.build_unet_maps(_dev(coords), levels), unet.build_unet_maps_host(coords, levels))


def test_rows_in_any_order():
    """Input rows keep the caller's order: the pairs of a shuffled cloud are those of the sorted one, renumbered."""
    from fgms_b200 import gpu_maps, maps
    coords = clouds.surface_cloud(5000, 64, 9)
    order = np.random.default_rng(1).permutation(coords.shape[0])
    shuffled = np.ascontiguousarray(coords[order])
    _same(gpu_maps.build_submanifold_map(_dev(shuffled), 3), maps.build_submanifold_map(shuffled, 3))
    _same(gpu_maps.build_strided_map(_dev(shuffled), 2), maps.build_strided_map(shuffled, 2, 2))


def test_memory_left_behind_by_an_earlier_cloud_does_not_matter():
    for seed in range(4):
        coords = clouds.uniform_cloud(3000 + 700 * seed, 30, seed)
        _check(unet.build_unet_maps(_dev(coords), 2), unet.build_unet_maps_host(coords, 2))


def test_every_map_has_memory_of_its_own():
    """A map that is kept does not keep the others, and an edit of one is no edit of what a backward has saved of another."""
    m = unet.build_unet_maps(_dev(np.unique(clouds.surface_cloud(5000, 64, 9), axis=0)), 2)
    maps = m.subm + m.down + m.up
    assert len({k.imap.untyped_storage().data_ptr() for k in maps}) == len(maps)
    before = [k.imap._version for k in maps]
    maps[0].imap[:1] = maps[0].imap[:1].clone()
    assert [k.imap._version for k in maps[1:]] == before[1:]


def test_counts_of_more_blocks_of_rows_than_a_warp_keeps():
    """A warp keeps the counts of 512 blocks of 256 rows: 131 072 rows.  175 616 are read again, 16 384 at a time."""
    coords = _block(56, 56, 56)
    _check(unet.build_unet_maps(_dev(coords), 1), unet.build_unet_maps_host(coords, 1))


@pytest.mark.parametrize("levels,what", [(1, 1), (3, 7), (5, 6)])
def test_sizes_in_memory_that_is_not_page_locked(levels, what):
    """The kernel writes page-locked sizes itself; others, written by a copy, are the same, and so are kpos and the coordinates."""
    coords = _dev(np.unique(clouds.surface_cloud(5000, 64, 9), axis=0))
    n, n_maps = coords.size(0), sum(levels - (kind > 1) for kind in (1, 2, 4) if what & kind)
    ws = torch.empty(_lib.lib.fgms_b200_pyramid_workspace_bytes(n, levels, what), dtype=torch.uint8, device="cuda")

    def plan(sizes_at):
        kpos = torch.zeros((n_maps, 28), dtype=torch.int32, device="cuda")
        coarser = [torch.zeros((n, 3), dtype=torch.int32, device="cuda") for _ in range(levels - 1)]
        at = (ctypes.c_void_p * max(1, levels - 1))(*[c.data_ptr() for c in coarser])
        _lib.check(_lib.lib.fgms_b200_pyramid_plan(coords.data_ptr(), n, levels, what, kpos.data_ptr(), at, ws.data_ptr(), ws.numel(), sizes_at,
                                                   torch.cuda.current_stream().cuda_stream))
        return [kpos] + coarser

    count = 1 + levels + n_maps
    locked, pageable = torch.full((count + 1,), 77, dtype=torch.int32, pin_memory=True), (ctypes.c_int32 * (count + 1))(*[77] * (count + 1))
    a, b = plan(locked.data_ptr()), plan(ctypes.addressof(pageable))
    assert locked.tolist() == list(pageable) and pageable[0] == 0 and pageable[1] == n and pageable[count] == 77
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    for j in range(n_maps):
        assert pageable[1 + levels + j] == int(a[0][j].max())
