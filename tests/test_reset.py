"""Reset: an emptied volume is a new one (no block, every slot empty, every
voxel zero), in each storage mode and table layout, whatever the number of
blocks it held (none, fewer than the reset kernel's CTAs, more)."""
from __future__ import annotations

import numpy as np
import pytest

from what_irregularity_costs_b200 import (CudaVolume, LAYOUT_POOL, LAYOUT_SLOT_INDEX, STORAGE_FP16_U16, STORAGE_FP32,
                                          STORAGE_FP64, device_tensor, scenes)

TYPES = {STORAGE_FP32: ("<f4", "<f4"), STORAGE_FP16_U16: ("<f2", "<i2"), STORAGE_FP64: ("<f8", "<f4")}


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [LAYOUT_POOL, LAYOUT_SLOT_INDEX])
@pytest.mark.parametrize("storage", [STORAGE_FP32, STORAGE_FP16_U16, STORAGE_FP64])
@pytest.mark.parametrize("size", [(8, 6), (160, 120)])
def test_reset_volume_is_a_new_one(cuda, storage, layout, size):
    K = scenes.ROOM_K.scaled(*size)
    frames = [scenes.room_frame(scenes.RoomScene.make(3), k, K) for k in range(2)]
    points = [cuda.from_numpy(scenes.frame_points(f)).cuda() for f in frames]
    vol = CudaVolume(0.03, 1 << 13, 0.12, 6.0, storage=storage, layout=layout)
    new = CudaVolume(0.03, 1 << 13, 0.12, 6.0, storage=storage, layout=layout)
    vol.reset()  # nothing allocated yet
    for p, f in zip(points, frames):
        vol.integrate(p, f.cam)
    assert vol.block_count() > 0
    vol.reset()
    assert vol.block_count() == 0 and vol.drop_count() == 0 and vol.status() == 0
    keys, idx = vol.table()
    assert np.all(keys == -1) and np.all(idx == -1)
    view = vol.device_view()
    for ptr, typ in zip((view.tsdf, view.weight), TYPES[storage]):
        assert int(cuda.count_nonzero(device_tensor(ptr, (view.pool_capacity, 512), typ))) == 0
    if storage == STORAGE_FP32:
        for ptr in (view.r, view.g, view.b):
            assert int(cuda.count_nonzero(device_tensor(ptr, (view.pool_capacity, 512), "<f4"))) == 0
    for v in (vol, new):
        for p, f in zip(points, frames):
            v.integrate(p, f.cam)
    # Read out by coordinate, in the arrays' own types (whole volumes, so that
    # both layouts read alike; slots in use have a key).
    out = []
    for v in (vol, new):
        v.synchronize()
        view = v.device_view()
        n = view.pool_capacity
        coords = device_tensor(view.block_coord, (n, 3), "<i4").cpu().numpy()
        if layout == LAYOUT_SLOT_INDEX:
            used = np.nonzero(v.table()[0] >= 0)[0]
        else:
            used = np.arange(v.block_count())
        used = used[np.lexsort(coords[used].T[::-1])]
        out.append([coords[used]] + [device_tensor(ptr, (n, 512), typ).cpu().numpy()[used]
                                     for ptr, typ in zip((view.tsdf, view.weight), TYPES[storage])])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
