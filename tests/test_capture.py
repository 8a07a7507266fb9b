"""Updates recorded by a stream capture: updates that run outside the graph
start from cleared counters whether the graph was launched or not, and a reset
leaves nothing of a graph's launches behind."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import sorted_voxels
from what_irregularity_costs_b200 import CudaVolume, scenes

CAP = 5.0


def _frames(cuda):
    K = scenes.ROOM_K.scaled(121, 77)
    room = scenes.RoomScene.make(5)
    frames = [scenes.room_frame(room, k, K) for k in range(3)]
    return [(cuda.from_numpy(scenes.frame_points(f)).cuda(), f.cam) for f in frames]


def _volume(frames):
    vol = CudaVolume(0.03, 1 << 13, 0.12, CAP)
    vol.integrate(*max(frames, key=lambda f: f[0].shape[0]))  # grows the records
    vol.reset()
    return vol


def _capture(cuda, vol, frame):
    graph, stream = cuda.cuda.CUDAGraph(), cuda.cuda.ExternalStream(vol.stream_handle())
    with cuda.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        vol.integrate(*frame)

    def launch():
        with cuda.cuda.stream(stream):
            graph.replay()
        vol.synchronize()
    return launch


def _plain(frames, which):
    """Map and per-update statistics of these frames, one after the other."""
    vol = _volume(frames)
    stats = []
    for k in which:
        vol.integrate(*frames[k])
        stats.append(vol.last_update_stats())
    return sorted_voxels(vol), stats


def _assert_same(vol, voxels):
    assert vol.status() == 0
    for a, b in zip(sorted_voxels(vol), voxels):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("before", [[], [0], [0, 1]])
@pytest.mark.parametrize("launches", [0, 1])
def test_updates_around_a_capture(cuda, launches, before):
    frames = _frames(cuda)
    vol = _volume(frames)
    for k in before:
        vol.integrate(*frames[k])
    launch = _capture(cuda, vol, frames[1])
    for _ in range(launches):
        launch()
    got = []
    for k in (2, 0, 2):
        vol.integrate(*frames[k])
        got.append(vol.last_update_stats())
    voxels, stats = _plain(frames, before + [1] * launches + [2, 0, 2])
    assert got == stats[-3:] and max(s["crossing_voxels"] for s in stats) > 0
    _assert_same(vol, voxels)


@pytest.mark.gpu
def test_reset_after_launches(cuda):
    """The second launch in a row leaves counts in voxels that no update
    finishes; a reset clears them."""
    frames = _frames(cuda)
    vol = _volume(frames)
    launch = _capture(cuda, vol, frames[1])
    for _ in range(2):
        launch()
    vol.reset()
    vol.integrate(*frames[1])
    vol.integrate(*frames[0])
    voxels, _ = _plain(frames, [1, 0])
    _assert_same(vol, voxels)
