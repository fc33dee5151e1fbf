"""The metrics kernel's launch shapes and the device's stone width: a pose scores the same in
a launch of any size, and degenerate plane sets score as the CPU oracle scores them."""
import math

import numpy as np
import pytest

from indicatrix_b200 import geometry, materials, workloads
from indicatrix_b200.backend import MetricsLighting

pytestmark = pytest.mark.gpu
LIGHT = MetricsLighting(10, 0.85, 0.95)


# 4 to 128 warps a pose: the last pose count of each shape and the first of the next.
@pytest.mark.parametrize("n", [2, 18, 19, 37, 38, 74, 75, 148, 149, 296, 297, 593])
@pytest.mark.parametrize("fire", [False, True])
def test_a_pose_scores_the_same_in_any_launch(exact_backend, n, fire):
    spec = workloads.random_stones(1, seed=n)[0]
    stone = (spec.planes, spec.material.dispersion)
    rng = np.random.default_rng(n)
    poses = [(0, float(rng.uniform(0.0, 6.28)), float(rng.uniform(0.3, 1.57))) for _ in range(n)]
    got = exact_backend.evaluate_metrics_batch([stone], poses, LIGHT, fire)
    for i in (0, n // 2, n - 1):
        alone = exact_backend.evaluate_metrics_batch([stone], [poses[i]], LIGHT, fire)
        assert np.array_equal(got[i], alone[0])


def box(sx, sy, sz):
    rows = []
    for axis, half in enumerate((sx, sy, sz)):
        for sign in (1.0, -1.0):
            n = [0.0, 0.0, 0.0]
            n[axis] = sign
            rows.append(n + [-half])
    return np.array(rows, np.float32)


@pytest.mark.parametrize("planes", [box(0.5, 0.3, 0.4), box(0.2, 0.3, 0.6), np.repeat(box(0.5, 0.3, 0.4), 3, axis=0),
                                    box(0.5, 0.3, 0.4)[:4], box(0.5, 0.3, 0.4)[:1],
                                    geometry.to_f32(geometry.step_cut())],
                         ids=["box", "narrow-x", "duplicates", "open", "half-space", "step"])
def test_stone_width_of_unusual_stones(exact_backend, oracle, planes):
    mat = materials.diamond()
    got = exact_backend.evaluate_gem_optical_metrics(planes, mat, 0.6, 1.1, LIGHT)
    want = oracle.metrics(planes, mat, 0.6, 1.1, LIGHT.preset, LIGHT.light_yaw, LIGHT.light_pitch,
                          LIGHT.head_shadow_deg)
    # All but fire, whose angle's arc cosine rounds apart, are the oracle's bits.
    for k in (0, 2, 3, 4):
        assert got[k].view(np.uint32) == np.float32(want[k]).view(np.uint32), (k, got, want)
    assert math.isclose(got[1], want[1], rel_tol=1e-5)
