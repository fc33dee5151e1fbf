"""The interior scan (reciprocal keys, one exact quotient) against the exact
slab scan: the same facet and the same bits of t wherever the ray starts."""
import ctypes as C

import numpy as np
import pytest

from indicatrix_b200 import geometry, materials, workloads
from indicatrix_b200.backend import FrameScene, camera_new

pytestmark = pytest.mark.gpu
CHECK_INTERIOR_HIT = 18


def prism(n):
    """n half-spaces: a ring of n - 2 sides and two caps (fewer than 3: what there is)."""
    rows = [[0.0, 1.0, 0.0, -0.4], [0.0, -1.0, 0.0, -0.3]][:n]
    for i in range(max(0, n - 2)):
        a = 2.0 * np.pi * i / (n - 2)
        rows.append([np.cos(a), 0.0, np.sin(a), -0.5])
    return np.array(rows, np.float32)


def rays(planes, rng, n):
    """Interior and exterior origins, origins on facets and a restart past them, rays along
    the axes, and rays at the prism's edges (two facets at one distance)."""
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[: n // 8] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, n // 8)] * rng.choice([-1.0, 1.0], (n // 8, 1)).astype(np.float32)
    o = rng.uniform(-0.3, 0.3, (n, 3)).astype(np.float32)
    o[n // 2: 5 * n // 8] = 0.0
    o[5 * n // 8: 3 * n // 4] *= np.float32(6.0)
    k = rng.integers(0, len(planes), n - 3 * n // 4)
    p = planes[k]
    side = np.einsum("ij,ij->i", o[3 * n // 4:], p[:, :3]) + p[:, 3]
    o[3 * n // 4:] -= (side[:, None] * p[:, :3]).astype(np.float32)
    o[7 * n // 8:] += np.float32(1e-4) * d[7 * n // 8:]
    return o, d


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 121, 127, 128, "brilliant", "step"])
def test_interior_scan_equals_the_exact_scan(exact_backend, backend, oracle, n):
    planes = {"brilliant": lambda: geometry.to_f32(geometry.round_brilliant()),
              "step": lambda: geometry.to_f32(geometry.step_cut())}.get(n, lambda: prism(n).reshape(-1, 4))()
    fs = FrameScene(camera_new(0.0, 1.0, 1.6, 42.0), 32, 32, planes, materials.diamond(), 32,
                    workloads.iso_hemisphere())
    o, d = rays(planes, np.random.default_rng(5), 4096)
    inp = np.zeros((2 * len(o), 7), np.uint32)
    inp[:, :3] = np.tile(o, (2, 1)).view(np.uint32)
    inp[:, 3:6] = np.tile(d, (2, 1)).view(np.uint32)
    inp[len(o):, 6] = 1
    for b in (exact_backend, backend):
        out = b.debug_check(fs, CHECK_INTERIOR_HIT, inp, 2)
        assert np.array_equal(out[: len(o)], out[len(o):])
    out = exact_backend.debug_check(fs, CHECK_INTERIOR_HIT, inp, 2).view(np.float32)[len(o):]
    t, f = C.c_float(), C.c_int32()
    for oo, dd, r in zip(o[::4], d[::4], out[::4]):
        hit = oracle.lib().ixo_intersect(oracle._f32p(planes), planes.shape[0], oracle._f32p(oo.copy()),
                                         oracle._f32p(dd.copy()), C.byref(t), C.byref(f))
        assert int(r[1]) == (f.value if hit else -1)
        if hit:
            assert r[0].view(np.uint32) == np.float32(t.value).view(np.uint32)
