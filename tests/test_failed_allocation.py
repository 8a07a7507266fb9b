"""An allocation that fails is that call's failure alone: volumes that exist
keep working, with no later call taking the error for its own."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import canonical_triangles, sorted_voxels
from what_irregularity_costs_b200 import CudaVolume, scenes


def _failing_create(cuda):
    free, _ = cuda.cuda.mem_get_info()
    hog = cuda.empty(max(free - 40 * 10**9, 0), dtype=cuda.uint8, device="cuda")
    with pytest.raises(Exception):
        CudaVolume(0.02, 1 << 22, 0.08, 64.0)  # 69 GB
    del hog
    cuda.cuda.empty_cache()


@pytest.mark.gpu
def test_calls_after_a_failed_creation(cuda):
    frame = scenes.room_frame(scenes.RoomScene.make(5), 0, scenes.ROOM_K.scaled(121, 77))
    points = cuda.from_numpy(scenes.frame_points(frame)).cuda()
    vol, plain = (CudaVolume(0.03, 1 << 13, 0.12, 0.0) for _ in range(2))
    plain.integrate(points, frame.cam)
    vol.integrate(points, frame.cam)
    want, mesh = sorted_voxels(plain), canonical_triangles(plain.extract_mesh(1 << 20))
    calls = {
        "reset": lambda: (vol.reset(), vol.integrate(points, frame.cam)),
        "extract": lambda: canonical_triangles(vol.extract_mesh(1 << 20)),
        "snapshot": lambda: vol.restore(vol.snapshot()),
        "integrate": lambda: (vol.integrate(points, frame.cam), vol.reset(), vol.integrate(points, frame.cam)),
    }
    for name, call in calls.items():
        _failing_create(cuda)
        call()
        assert vol.status() == 0, name
        for a, b in zip(sorted_voxels(vol), want):
            assert np.array_equal(a, b), name
    assert np.array_equal(canonical_triangles(vol.extract_mesh(1 << 20)), mesh)


@pytest.mark.gpu
def test_pipelined_calls_after_scratch_that_did_not_fit(cuda):
    """Memory for the first scratch set of a large call but not for the second:
    the call fails, and smaller ones allocate both again."""
    frame = scenes.room_frame(scenes.RoomScene.make(5), 0, scenes.ROOM_K.scaled(121, 77))
    points = cuda.from_numpy(scenes.frame_points(frame)).cuda()
    many = cuda.zeros((14_000_000, 3), dtype=cuda.float32, device="cuda")
    vol, plain = (CudaVolume(0.03, 1 << 13, 0.12, 3.0) for _ in range(2))
    vol.set_pipelined(True)
    vol.integrate(points, frame.cam)
    vol.synchronize()
    cuda.cuda.empty_cache()
    hog = cuda.empty(cuda.cuda.mem_get_info()[0] - 2_200_000_000, dtype=cuda.uint8, device="cuda")
    # A band slot takes 18 bytes in the first set and 8 in the second.
    n = cuda.cuda.mem_get_info()[0] // 22 // 9
    assert 1_000_000 < n <= many.shape[0]
    with pytest.raises(RuntimeError):
        vol.integrate(many, frame.cam, 0.0, n)
    del hog
    cuda.cuda.empty_cache()
    plain.integrate(points, frame.cam)
    for _ in range(4):
        vol.integrate(points, frame.cam)
        plain.integrate(points, frame.cam)
    vol.synchronize()
    assert vol.status() == 0
    for a, b in zip(sorted_voxels(vol), sorted_voxels(plain)):
        assert np.array_equal(a, b)
