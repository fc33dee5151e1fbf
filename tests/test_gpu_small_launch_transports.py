"""The path pool's claims of four paths, on every transport and in both builds: samples traced one
launch each (claims of four) add up to the sums of one launch of them all (claims of 32)."""
import numpy as np
import pytest

from indicatrix_b200 import abi, materials, workloads
from indicatrix_b200.backend import GpuBackend

pytestmark = pytest.mark.gpu
POOL_MIDDLE_BUDGET = 4  # budget + 3 * shape: the 128-thread pool at the middle register budget
WIDTH, HEIGHT, SPP = 80, 64, 64  # 5120 and 327,680 paths: below and above 64 a resident warp


def biaxial(w, h):
    fs = workloads.round_brilliant_frame(w, h, max_bounces=24)
    fs.material = materials.topaz((0.3, 0.8, 0.52))
    return fs


@pytest.mark.parametrize("precision", [abi.PRECISION_EXACT, abi.PRECISION_FAST], ids=["exact", "fast"])
@pytest.mark.parametrize("make", [workloads.round_brilliant_frame, workloads.anisotropic_stress_frame,
                                  workloads.carved_sun_frame, biaxial],
                         ids=["isotropic", "uniaxial", "sun", "biaxial"])
def test_launches_of_one_sample_add_up(make, precision):
    b = GpuBackend.acquire(precision=precision, kernel_variant=POOL_MIDDLE_BUDGET + 1)
    fs = make(WIDTH, HEIGHT)
    parts, whole = np.zeros((2, HEIGHT, WIDTH, 3))
    for s in range(SPP):
        assert b.try_accumulate(fs, 9 + s, 1, parts)
    assert b.try_accumulate(fs, 9, SPP, whole)
    b.close()
    assert whole.max() > 0.0
    # The same non-negative samples: one f64 rounding a launch and one an addition.
    assert np.all(np.abs(parts - whole) <= 2 * SPP * np.finfo(np.float64).eps * whole)
