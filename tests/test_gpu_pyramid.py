"""The pyramid builder (``csrc/map_pyramid.cuh``): every map of every level equals the host builders' bit for bit, for rows
in any order, boxes around the 32-cell words of its bitmaps, and clouds it has to leave to the hash-table builders."""
import numpy as np
import pytest
import torch

from fgms_b200 import clouds, unet
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
