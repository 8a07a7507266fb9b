"""last_update_stats after batched steps, whatever serial updates came before
them: each update's statistics are those of the same call on a volume that
has its counters to itself, with voxels that cross the cap among them."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import sorted_voxels
from what_irregularity_costs_b200 import Batch, CudaVolume, scenes

VOXEL, CAP, POOL = 0.03, 5.0, 1 << 13


@pytest.mark.gpu
@pytest.mark.parametrize("n_serial", [0, 1, 2, 3])
def test_statistics_of_batched_steps(cuda, n_serial):
    K = scenes.ROOM_K.scaled(121, 77)
    room = scenes.RoomScene.make(5)
    frames = [scenes.room_frame(room, k, K) for k in range(6)]
    points = [cuda.from_numpy(scenes.frame_points(f)).cuda() for f in frames]

    def alone(upto):
        """Statistics and map of frames 0 .. upto, each the first update after
        its volume was pipelined anew: a control block of its own, cleared."""
        vol = CudaVolume(VOXEL, POOL, 4 * VOXEL, CAP)
        for k in range(upto + 1):
            vol.set_pipelined(True)
            vol.integrate(points[k], frames[k].cam)
            stats = vol.last_update_stats()
            vol.set_pipelined(False)
        return stats, sorted_voxels(vol)

    vol, other = (CudaVolume(VOXEL, POOL, 4 * VOXEL, CAP) for _ in range(2))
    for k in range(n_serial):
        vol.integrate(points[k], frames[k].cam)
    batch = Batch(2)
    most = max(p.shape[0] for p in points)
    batch.add(vol, most)
    batch.add(other, most)
    k = n_serial
    for idle in (False, True, False):
        # An idle scene keeps the statistics of its last update.
        if not idle:
            batch.set_frame(0, points[k], frames[k].cam)
            k += 1
        batch.set_frame(1, points[0], frames[0].cam)
        batch.step()
        batch.synchronize()
        want, _ = alone(k - 1)
        assert vol.last_update_stats() == want, (n_serial, idle)
    vol.integrate(points[k], frames[k].cam)
    want, voxels = alone(k)
    assert vol.last_update_stats() == want and want["crossing_voxels"] > 0
    for a, b in zip(sorted_voxels(vol), voxels):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_idle_scene_keeps_serial_statistics(cuda):
    """A batched step that leaves a scene out does not replace what its last
    serial update counted, in either of its control blocks."""
    K = scenes.ROOM_K.scaled(121, 77)
    frame = scenes.room_frame(scenes.RoomScene.make(5), 0, K)
    points = cuda.from_numpy(scenes.frame_points(frame)).cuda()
    vol, other = (CudaVolume(VOXEL, POOL, 4 * VOXEL, CAP) for _ in range(2))
    batch = Batch(2)
    batch.add(vol, points.shape[0])
    batch.add(other, points.shape[0])
    for _ in range(3):
        vol.integrate(points, frame.cam)
        want = vol.last_update_stats()
        batch.set_frame(1, points, frame.cam)
        batch.step()
        batch.synchronize()
        assert vol.last_update_stats() == want
