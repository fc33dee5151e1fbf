"""The interior scan on rays at a stone's vertices and edges, where two or more planes lie at one
distance or a few units of 2^-16 apart, and on stones with doubled planes: the exact scan's facet
and the bits of its t."""
import itertools

import numpy as np
import pytest

from indicatrix_b200 import geometry, materials, workloads
from indicatrix_b200.backend import FrameScene, camera_new

pytestmark = pytest.mark.gpu
CHECK_INTERIOR_HIT = 18


def box():
    rows = [[s * (a == 0), s * (a == 1), s * (a == 2), -h] for a, h in enumerate((0.5, 0.3, 0.4)) for s in (1.0, -1.0)]
    return np.array(rows, np.float32)


def stone(name):
    return {"box": box, "step": lambda: geometry.to_f32(geometry.step_cut()),
            "brilliant": lambda: geometry.to_f32(geometry.round_brilliant()),
            "box x 3": lambda: np.repeat(box(), 3, axis=0),
            "step x 2": lambda: np.tile(geometry.to_f32(geometry.step_cut()), (2, 1))}[name]()


def corners(planes):
    """Vertices of the solid in f64 (up to 4000 of them) with the distinct planes through each."""
    p = np.unique(planes.astype(np.float64), axis=0)
    tri = np.array(list(itertools.combinations(range(len(p)), 3)))
    if len(tri) > 60000:
        tri = tri[np.random.default_rng(0).permutation(len(tri))[:60000]]
    n = p[tri][:, :, :3]
    ok = np.abs(np.linalg.det(n)) > 1e-6
    v = np.linalg.solve(n[ok], -p[tri[ok]][:, :, 3:])[:, :, 0]
    keep = (v @ p[:, :3].T + p[:, 3]).max(axis=1) < 1e-6
    return v[keep][:4000], tri[ok][keep][:4000]


def targets(planes, rng, n):
    v, t = corners(planes)
    a = rng.integers(0, len(v), n)
    out = v[a].copy()
    # Half of them on an edge: between the vertex and another on two of its planes.
    for i in range(0, n, 2):
        near = [j for j in rng.permutation(len(v))[:200] if len(set(t[j]) & set(t[a[i]])) == 2]
        if near:
            out[i] += rng.uniform(0.1, 0.9) * (v[near[0]] - v[a[i]])
    return out


@pytest.mark.parametrize("name", ["box", "step", "brilliant", "box x 3", "step x 2"])
def test_rays_at_edges_and_vertices(exact_backend, backend, name):
    planes, rng, n = stone(name), np.random.default_rng(11), 4096
    at = targets(planes, rng, n)
    o = rng.uniform(-0.12, 0.12, (n, 3)) * [1.0, 0.5, 1.0]
    shift = rng.choice([0.0] + [2.0 ** -e for e in range(14, 21)], (n, 1)) * rng.choice([-1.0, 1.0], (n, 3))
    d = at * (1.0 + shift) - o
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = o.astype(np.float32)
    # What the stone is for: many rays whose two nearest distinct planes are closer than the
    # scan's keys can tell.
    u = np.unique(planes.astype(np.float64), axis=0)
    key = np.sort((d @ u[:, :3].T) / (o @ u[:, :3].T + u[:, 3]), axis=1)
    assert np.all(o @ planes[:, :3].T + planes[:, 3] < 0)
    assert np.sum(key[:, 1] <= key[:, 0] * (1.0 - 2.0 ** -16)) > n // 8
    inp = np.zeros((2 * n, 7), np.uint32)
    inp[:, :3] = np.tile(o, (2, 1)).view(np.uint32)
    inp[:, 3:6] = np.tile(d, (2, 1)).view(np.uint32)
    inp[n:, 6] = 1
    fs = FrameScene(camera_new(0.0, 1.0, 1.6, 42.0), 32, 32, planes, materials.diamond(), 32,
                    workloads.iso_hemisphere())
    for b in (exact_backend, backend):
        out = b.debug_check(fs, CHECK_INTERIOR_HIT, inp, 2)
        assert np.array_equal(out[:n], out[n:])
