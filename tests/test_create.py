"""Creating a volume takes the same time whatever its truncation distance."""
import time

import pytest

from what_irregularity_costs_b200 import CudaVolume


@pytest.mark.gpu
def test_long_truncation_is_created_at_once(cuda):
    def create(trunc):
        times = []
        for _ in range(3):
            t0 = time.perf_counter()
            vol = CudaVolume(1e-3, 64, trunc, 0.0)
            times.append(time.perf_counter() - t0)
            assert vol.block_count() == 0
        return min(times)

    create(0.004)
    # 2e9 band steps: one by one they take seconds; a volume, milliseconds.
    assert create(2e6) < create(0.004) + 0.25
