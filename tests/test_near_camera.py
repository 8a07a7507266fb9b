"""Points closer to the camera than their band is long: samples before the
camera's far side lie behind it and may be fully occluded, which the oracle
rejects (blocks and weights exact, mean TSDF within the parity bar)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import FP16_ORACLE_TOL, TSDF_TOL, assert_matches_oracle
from what_irregularity_costs_b200 import (STORAGE_FP16_U16, STORAGE_FP32, STORAGE_FP64, Batch, CudaVolume)

VOXEL = 0.02
CAM = (0.313, -0.207, 0.118)


def cloud(seed=0, n=4000):
    """Points 0.05 to 12 voxels from the camera, most of them within one."""
    rng = np.random.default_rng(seed)
    d = rng.standard_normal((n, 3))
    r = VOXEL * np.where(np.arange(n) % 4 < 3, rng.uniform(0.05, 1.0, n), rng.uniform(1.0, 12.0, n))
    return (np.asarray(CAM) + r[:, None] * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _integrate(vol, d):
    vol.integrate(d, CAM)


def _split(vol, d):
    vol.allocate_blocks(d, CAM)
    vol.update_voxels(d, CAM)


def _frames(vol, d):
    n = d.shape[0]
    vol.integrate_frames(d, np.array([0, n // 3, n], dtype=np.int32), [CAM, CAM])


def _batch(vol, d):
    batch = Batch(1)
    batch.add(vol, d.shape[0])
    batch.set_frame(0, d, CAM)
    batch.step()
    batch.remove(0)


PATHS = {
    "integrate": (STORAGE_FP32, _integrate, TSDF_TOL),
    "two stages": (STORAGE_FP32, _split, TSDF_TOL),
    "several frames": (STORAGE_FP32, _frames, TSDF_TOL),
    "batch": (STORAGE_FP32, _batch, TSDF_TOL),
    "fp16": (STORAGE_FP16_U16, _integrate, FP16_ORACLE_TOL),
    "fp64": (STORAGE_FP64, _integrate, TSDF_TOL),
}


def test_oracle_rejects_samples_behind_the_camera():
    """The cloud holds what the test is about: near points lose samples."""
    points = cloud()
    for trunc in (2.1, 4.0, 6.5):
        ref = oracle.OracleVolume(VOXEL, 1 << 12, trunc * VOXEL, 0.0)
        ref.integrate(points, CAM)
        steps = int(np.ceil(np.float32(np.float32(trunc * VOXEL) * (np.float32(1.0) / np.float32(VOXEL)))))
        assert ref.voxels()[2].sum() < points.shape[0] * (2 * steps + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [6.0, 0.0])
@pytest.mark.parametrize("trunc", [2.1, 4.0, 6.5])
@pytest.mark.parametrize("path", list(PATHS))
def test_near_points_match_oracle(cuda, path, trunc, cap):
    storage, call, tol = PATHS[path]
    points = cloud()
    vol = CudaVolume(VOXEL, 1 << 12, trunc * VOXEL, cap, storage=storage)
    ref = oracle.OracleVolume(VOXEL, 1 << 12, trunc * VOXEL, cap)
    call(vol, cuda.from_numpy(points).cuda())
    ref.integrate(points, CAM)
    assert vol.status() == 0 and vol.drop_count() == 0
    assert_matches_oracle(vol, ref, tol)
