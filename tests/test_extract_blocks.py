"""Extraction where a block's list, the row bits and the aligned copy-out end:
noise volumes whose blocks emit thousands of triangles, single blocks, thin
valid layers, against the CPU oracle triangle for triangle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import assert_same_voxels, canonical_triangles
from what_irregularity_costs_b200 import CudaVolume, LAYOUT_POOL, LAYOUT_SLOT_INDEX


def noise(n, extent, seed):
    """Points all over a cube, seen from a camera within it: SDF signs at random."""
    return (np.random.default_rng(seed).uniform(-extent, extent, (n, 3)) + 0.017).astype(np.float32)


CASES = {
    # name: (points, camera, voxel, truncation in voxels)
    "dense blocks": (noise(60000, 0.3, 1), (0.013, 0.007, -0.011), 0.02, 2.0),
    "one dense block": (noise(20000, 0.06, 2) + np.float32(0.08), (0.5, 0.4, 0.3), 0.02, 1.0),
    "sparse": (noise(300, 0.4, 3), (2.0, 0.3, 0.1), 0.02, 4.0),
    "one point": (noise(1, 0.1, 4), (0.9, 0.2, 0.3), 0.02, 4.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [LAYOUT_POOL, LAYOUT_SLOT_INDEX])
@pytest.mark.parametrize("name", list(CASES))
def test_mesh_matches_oracle(cuda, name, layout):
    points, cam, voxel, trunc = CASES[name]
    # Cap 1: every voxel takes one contribution, so both volumes are bit-identical.
    vol = CudaVolume(voxel, 1 << 10, trunc * voxel, 1.0, layout=layout)
    ref = oracle.OracleVolume(voxel, 1 << 10, trunc * voxel, 1.0)
    vol.integrate(cuda.from_numpy(points).cuda(), cam)
    ref.integrate(points, cam)
    assert_same_voxels(vol, ref, exact_tsdf=True)
    want = ref.extract(0.5, 0.0, 1 << 22)
    cap = want.shape[0] + 8
    buf = cuda.full((cap * 6 + 8,), 7.0, dtype=cuda.float32, device="cuda")
    for pad in (0, 1, 3):  # the output buffer need not be 16-byte aligned
        buf.fill_(7.0)
        n = vol.extract_mesh_device(buf.data_ptr() + 4 * pad, vert_cap=cap)
        assert n == want.shape[0]
        got = buf.cpu().numpy()
        assert np.all(got[:pad] == 7.0) and np.all(got[pad + 6 * n:] == 7.0)
        mesh = got[pad:pad + 6 * n].reshape(-1, 6)
        assert np.array_equal(canonical_triangles(mesh), canonical_triangles(want))
    if name == "dense blocks":
        assert want.shape[0] // 3 > 1024 * vol.block_count()  # several lists per block
    if want.shape[0]:
        assert vol.extract_mesh_device(buf.data_ptr(), vert_cap=want.shape[0] - 1) == -1  # overflow
        rgb = cuda.full((cap * 3 + 4,), 9, dtype=cuda.uint8, device="cuda")
        for pad in (0, 1, 2):
            rgb.fill_(9)
            assert vol.extract_mesh_device(buf.data_ptr(), rgb.data_ptr() + pad, cap) == want.shape[0]
            col = rgb.cpu().numpy()
            assert np.all(col[pad:pad + 3 * n] == 128) and np.all(np.delete(col, np.s_[pad:pad + 3 * n]) == 9)
