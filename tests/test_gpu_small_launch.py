"""Launches that the path pool claims in quads, and those just past that: the same sums as
the static task loop's (the exact build: both add the same samples)."""
import numpy as np
import pytest

from indicatrix_b200 import abi, workloads
from indicatrix_b200.backend import GpuBackend

pytestmark = pytest.mark.gpu
VARIANT_TASKS = 2  # the task loop under the second occupancy budget


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (3, 1, 1), (2, 2, 1), (5, 1, 1), (7, 3, 5), (160, 120, 1),
                                              (592, 511, 1), (592, 512, 1), (592, 513, 1)])
def test_small_launches_add_the_same_samples(exact_backend, width, height, spp):
    tasks = GpuBackend.acquire(precision=abi.PRECISION_EXACT, kernel_variant=VARIANT_TASKS + 1)
    fs = workloads.round_brilliant_frame(width, height)
    got, want = np.zeros((2, height, width, 3))
    assert exact_backend.try_accumulate(fs, 3, spp, got) and tasks.try_accumulate(fs, 3, spp, want)
    tasks.close()
    # Sums of at most 5 non-negative f32 samples: f64 rounding alone.
    assert np.all(np.abs(got - want) <= 4 * np.finfo(np.float64).eps * np.abs(want) + 1e-15)
