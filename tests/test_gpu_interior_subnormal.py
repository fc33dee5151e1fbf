"""The interior scan from origins closer to a facet than the smallest normal number: the exact
scan's answer, though the facet's reciprocal overflows."""
import numpy as np
import pytest

from indicatrix_b200 import materials, workloads
from indicatrix_b200.backend import FrameScene, camera_new

pytestmark = pytest.mark.gpu
CHECK_INTERIOR_HIT = 18


@pytest.mark.parametrize("at", [0, 1, 5])
def test_origin_a_subnormal_distance_inside_a_facet(exact_backend, backend, at):
    # A box whose floor passes through the origin of the coordinates, so that a ray's distance
    # from it can be any float; the floor is plane `at`.
    planes = [[0.0, 1.0, 0.0, -0.4], [1.0, 0.0, 0.0, -0.5], [-1.0, 0.0, 0.0, -0.5], [0.0, 0.0, 1.0, -0.5],
              [0.0, 0.0, -1.0, -0.5]]
    planes.insert(at, [0.0, -1.0, 0.0, 0.0])
    planes = np.array(planes, np.float32)
    rng = np.random.default_rng(at)
    heights = [1e-45, 1e-44, 1e-42, 1e-40, 5e-39, 1.1e-38, 1.2e-38, 1e-36, 1e-30, 1e-25, 1e-20, 1e-15, 1e-10, 0.0]
    o = rng.uniform(-0.4, 0.4, (len(heights) * 16, 3)).astype(np.float32)
    o[:, 1] = np.repeat(np.array(heights, np.float32), 16)
    d = rng.normal(size=o.shape).astype(np.float32)
    d[::2, 1] = -np.abs(d[::2, 1])  # half of them towards the floor
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    inp = np.zeros((2 * len(o), 7), np.uint32)
    inp[:, :3] = np.tile(o, (2, 1)).view(np.uint32)
    inp[:, 3:6] = np.tile(d, (2, 1)).view(np.uint32)
    inp[len(o):, 6] = 1
    fs = FrameScene(camera_new(0.0, 1.0, 1.6, 42.0), 32, 32, planes, materials.diamond(), 32,
                    workloads.iso_hemisphere())
    for b in (exact_backend, backend):
        out = b.debug_check(fs, CHECK_INTERIOR_HIT, inp, 2)
        assert np.array_equal(out[: len(o)], out[len(o):])
