"""The band walk where its warp table, its float shortcuts and its limits end:
each cloud against the CPU oracle (blocks, weights and colours exact, mean
TSDF within the parity bar)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import assert_same_blocks, assert_same_voxels
from what_irregularity_costs_b200 import CudaVolume, scenes


def sphere(n=1500, radius=0.5, centre=(0.0, 0.0, 2.0), seed=0):
    d = np.random.default_rng(seed).standard_normal((n, 3))
    return (np.asarray(centre) + radius * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def interleaved(n_clusters, gap):
    """Neighbouring points alternate between clusters `gap` metres apart."""
    parts = [sphere(400, 0.3, (gap * (k + 1), -gap * (k % 3), 0.5 * gap * (k % 2)), k) for k in range(n_clusters)]
    return np.stack(parts, 1).reshape(-1, 3)


def edge_rows():
    """Rows of points whose depth jumps by metres from pixel to pixel."""
    f = scenes.sphere_frame(scenes.Intrinsics(97, 31, 73.0, 73.0, 48.0, 15.0))
    z = np.where(f.depth > 0, f.depth, 6.0).astype(np.float32)
    z[:, ::5] *= np.float32(0.5)
    return scenes.backproject(z, f.K, f.R, f.t)


CLOUDS = {
    # name: (points, camera, voxel, truncation in voxels)
    "shuffled": (sphere(), (0.0, 0.0, 0.0), 0.02, 4.0),                     # entries that many blocks share
    "one point": (sphere(1), (0.0, 0.0, 0.0), 0.02, 4.0),
    "33 points": (sphere(33), (0.0, 0.0, 0.0), 0.01, 4.0),
    "depth edges": (edge_rows(), (0.0, 0.0, 0.0), 0.02, 4.0),
    "two clusters": (interleaved(2, 15.0), (0.0, 0.0, 0.0), 0.01, 4.0),     # a second round per warp
    "six clusters": (interleaved(6, 15.0), (1.0, 2.0, 3.0), 0.01, 4.0),     # sample by sample
    "400 m away": (sphere(900, 0.5, (400.0, -400.0, 380.0)), (399.0, -399.0, 379.0), 0.01, 4.0),
    "25 km away": (sphere(900, 2.0, (25000.0, -9000.0, 60.0)), (25004.0, -9003.0, 61.0), 0.01, 4.0),
    "three chunks": (sphere(900), (0.1, 0.0, -0.2), 0.01, 11.3),
    "long band": (sphere(40), (0.0, 0.0, 0.0), 0.004, 495.0),               # longer than the offsets hold
    "short band": (sphere(900), (0.0, 0.0, 0.0), 0.02, 0.4),
}


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [6.0, 0.0])
@pytest.mark.parametrize("name", list(CLOUDS))
def test_walk_matches_oracle(cuda, name, cap):
    points, cam, voxel, trunc = CLOUDS[name]
    vol = CudaVolume(voxel, 1 << 15, trunc * voxel, cap)
    ref = oracle.OracleVolume(voxel, 1 << 15, trunc * voxel, cap)
    d = cuda.from_numpy(points).cuda()
    vol.integrate(d, cam)
    vol.allocate_blocks(d, cam)
    vol.update_voxels(d, cam)
    for _ in range(2):
        ref.integrate(points, cam)
    assert vol.status() == 0 and vol.drop_count() == ref.drop_count() == 0
    assert_same_blocks(vol, ref)
    assert_same_voxels(vol, ref)


@pytest.mark.gpu
def test_walk_drops_where_the_pool_is_full(cuda):
    """Warps that meet dropped blocks: admitted voxels are the oracle's, and
    every sample is either in a voxel or counted as dropped."""
    points, cam = sphere(1200), (0.0, 0.0, 0.0)
    vol = CudaVolume(0.02, 40, 0.08, 0.0)
    full = oracle.OracleVolume(0.02, 1 << 12, 0.08, 0.0)
    vol.integrate(cuda.from_numpy(points).cuda(), cam)
    full.integrate(points, cam)
    coords, _, weight = vol.means()
    rc, _, rw, *_ = full.voxels()
    want = {tuple(c): w for c, w in zip(rc.tolist(), rw)}
    assert coords.shape[0] == 40
    for c, w in zip(coords.tolist(), weight):
        assert np.array_equal(w, want[tuple(c)])
    assert vol.drop_count() == int(rw.sum() - weight.sum())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 29, 257, 2051])
@pytest.mark.parametrize("cap", [1.0, 2.5, 5.0])
def test_every_record_crosses(cuda, n, cap):
    """Grouping where all 256 band slots of a warp belong to cap-crossing
    voxels, and where the slots end inside a thread's eight."""
    points = np.tile(np.array([[0.013, 0.021, 1.007]], dtype=np.float32), (n, 1))
    points[1::3, 0] += np.float32(0.3)
    vol = CudaVolume(0.02, 1 << 10, 0.08, cap)
    ref = oracle.OracleVolume(0.02, 1 << 10, 0.08, cap)
    vol.integrate(cuda.from_numpy(points).cuda(), (0.0, 0.0, 0.0))
    ref.integrate(points, (0.0, 0.0, 0.0))
    assert vol.status() == 0
    assert_same_voxels(vol, ref)
