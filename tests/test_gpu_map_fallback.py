"""Clouds the bitmap builder leaves to the hash-table builders: it is asked once, not once per map, and neither its
scratch nor the lack of it stands in the way of a cloud that the hash-table builders can do."""
import numpy as np
import pytest
import torch

from fgms_b200 import clouds, gpu_maps, unet
from tests.test_gpu_maps import _dev, _same
from tests.test_gpu_pyramid import _check

pytestmark = pytest.mark.gpu


class _Counting:
    """``_native`` with its pyramid calls counted."""

    def __init__(self, native):
        self._native, self.calls = native, 0

    def __getattr__(self, name):
        return getattr(self._native, name)

    def build_pyramid(self, *args):
        self.calls += 1
        return self._native.build_pyramid(*args)


def _batch(scenes, voxels=3000):
    parts = []
    for s in range(scenes):
        c = clouds.surface_cloud(voxels, 48, 30 + s).copy()
        c[:, 0] += 4096 * 8 * s
        c[:, 1] += 4096 * 8 * s
        parts.append(c)
    return np.unique(np.concatenate(parts), axis=0)


def test_a_batch_of_scenes_is_refused_once_and_built_right(monkeypatch):
    coords = _batch(4)
    counting = _Counting(gpu_maps._native)
    monkeypatch.setattr(gpu_maps, "_native", counting)
    got = unet.build_unet_maps(_dev(coords), 4)
    _check(got, unet.build_unet_maps_host(coords, 4))
    assert counting.calls == 1


@pytest.mark.parametrize("pitch", [200, 4096])
def test_a_batch_along_x_equals_the_host_builders(pitch):
    parts = []
    for s in range(3):
        c = clouds.surface_cloud(4000, 64, 50 + s).copy()
        c[:, 0] += pitch * s
        parts.append(c)
    coords = np.unique(np.concatenate(parts), axis=0)
    _check(unet.build_unet_maps(_dev(coords), 4), unet.build_unet_maps_host(coords, 4))


def test_a_voxel_met_twice_is_refused_once(monkeypatch):
    coords = clouds.uniform_cloud(1000, 20, 2)
    coords = np.concatenate([coords, coords[:3]])
    counting = _Counting(gpu_maps._native)
    monkeypatch.setattr(gpu_maps, "_native", counting)
    unet.build_unet_maps(_dev(coords), 3)
    assert counting.calls == 1


def test_a_small_cloud_takes_little_memory():
    coords = _dev(clouds.surface_cloud(300, 20, 5))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    gpu_maps.build_submanifold_map(coords, 3)
    gpu_maps.build_strided_map(coords, 2)
    assert torch.cuda.max_memory_allocated() - before < 2 << 20


def test_a_wide_box_without_room_for_its_bitmaps_is_still_built():
    """2000 x 2000 x 80 cells take 64 MB of bits; with 40 MB left the hash-table builders do it."""
    coords = np.unique(np.random.default_rng(3).integers(0, [2000, 2000, 80], (3000, 3)).astype(np.int32), axis=0)
    dev = _dev(coords)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (40 << 20)) / total)
        got = unet.build_unet_maps(dev, 2)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    _check(got, unet.build_unet_maps_host(coords, 2))
