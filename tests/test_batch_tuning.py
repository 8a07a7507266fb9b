"""The autotuner times each shape that differs once: four tile counts. The
inert parts of a shape are reported with the time of their tile count."""
from __future__ import annotations

import pytest

from what_irregularity_costs_b200 import Batch, CudaVolume, scenes


@pytest.mark.gpu
@pytest.mark.parametrize("steps_per_shape", [1, 3])
def test_tuning_takes_four_shapes(cuda, steps_per_shape):
    frame = scenes.room_frame(scenes.RoomScene.make(5), 0, scenes.ROOM_K.scaled(121, 77))
    points = cuda.from_numpy(scenes.frame_points(frame)).cuda()
    vol = CudaVolume(0.03, 1 << 13, 0.12, 0.0)
    batch = Batch(1)
    batch.add(vol, points.shape[0])
    batch.autotune(steps_per_shape)
    for k in range(4 * steps_per_shape):
        assert batch.shape()["tuning"], k
        batch.set_frame(0, points, frame.cam)
        batch.step()
    shape, results = batch.shape(), batch.tune_results()
    assert not shape["tuning"]
    times = {r["tiles_per_item"]: r["median_ms"] for r in results}
    assert sorted(times) == [1, 2, 4, 8] and min(times.values()) > 0
    assert len(results) == 16 and all(r["median_ms"] == times[r["tiles_per_item"]] for r in results)
    assert len({(r["tiles_per_item"], r["probe"], r["finish_pair"]) for r in results}) == 16
    assert times[shape["tiles_per_item"]] == min(times.values())
    assert batch.status() == 0


@pytest.mark.gpu
def test_shapes_of_a_replayed_step(cuda):
    """Shapes that differ in their inert parts share a captured step."""
    frame = scenes.room_frame(scenes.RoomScene.make(5), 0, scenes.ROOM_K.scaled(121, 77))
    points = cuda.from_numpy(scenes.frame_points(frame)).cuda()
    batched, alone = (CudaVolume(0.03, 1 << 13, 0.12, 4.0) for _ in range(2))
    batch = Batch(1)
    batch.add(batched, points.shape[0])
    batch.set_graph(True)
    for shape in [(4, 0, 1), (4, 0, 1), (4, 1, 0), (4, 0, 0), (2, 1, 1), (2, 0, 1)]:
        batch.set_shape(*shape)
        batch.set_frame(0, points, frame.cam)
        batch.step()
        alone.integrate(points, frame.cam)
        got = batch.shape()
        assert (got["tiles_per_item"], got["probe"], got["finish_pair"]) == (
            shape[0], ["warp", "lane"][shape[1]], bool(shape[2]))
    batch.synchronize()
    assert batched.last_update_stats() == alone.last_update_stats()
    assert batched.block_count() == alone.block_count() and batch.status() == 0
