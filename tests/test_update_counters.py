"""The control counters of an update start at zero whatever kind of update
came before it: every call's statistics are what it added to the map."""
from __future__ import annotations

import numpy as np
import pytest

from what_irregularity_costs_b200 import Batch, CudaVolume, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [0.0, 1e6])
def test_statistics_across_kinds_of_update(cuda, cap):
    K = scenes.ROOM_K.scaled(121, 77)
    room = scenes.RoomScene.make(5)
    frames = [scenes.room_frame(room, k, K) for k in range(3)]
    points = [cuda.from_numpy(scenes.frame_points(f)).cuda() for f in frames]
    vol = CudaVolume(0.03, 1 << 13, 0.12, cap)
    begin = np.cumsum([0] + [p.shape[0] for p in points]).astype(np.int32)
    weights = {}

    def added():
        """(records, touched blocks, updated voxels) since the last look."""
        coords, _, w = vol.means()
        out = [0, 0, 0]
        for c, row in zip(map(tuple, coords.tolist()), w):
            d = row - weights.get(c, 0.0)
            out = [out[0] + int(d.sum()), out[1] + int(d.any()), out[2] + int(np.count_nonzero(d))]
            weights[c] = row
        return out

    def batched():
        batch = Batch(2)
        batch.add(vol, points[0].shape[0] + points[1].shape[0])
        batch.set_frame(0, points[1], frames[1].cam)
        batch.step()
        batch.remove(0)

    def empty():  # no point passes the cutoff: nothing is added
        vol.integrate(points[0], frames[0].cam, 1e-3)

    one = lambda k: lambda: vol.integrate(points[k], frames[k].cam)  # noqa: E731
    calls = [one(0), one(1), lambda: vol.update_voxels_noalloc(points[0], frames[0].cam), one(2), empty, one(0), batched,
             one(1), lambda: vol.integrate_frames(cuda.cat(points), begin, [f.cam for f in frames]),
             lambda: vol.set_pipelined(True), one(0), one(1), one(2), lambda: vol.set_pipelined(False), one(1), one(0)]
    for i, call in enumerate(calls):
        call()
        records, touched, updated = added()
        if i in (9, 13):  # no update
            continue
        stats = vol.last_update_stats()
        assert (stats["records"], stats["touched_blocks"], stats["updated_voxels"]) == (records, touched, updated), i
        assert stats["crossing_voxels"] == 0
