"""The one-launch clustering build (k_ploc) at the edges of its tiles (1024 clusters), its cluster of 8 blocks and its
shared-memory tail: closest hits through the tree against the segment test over every triangle (lighter_math.cpp:315-354
in FP32 with the same order of operations: equal bit for bit, since hits do not depend on the tree), runs of equal
boxes, a topology check of whole bakes, and a soup whose boxes have no order."""
import numpy as np
import pytest

from lighter_gb300 import ext, scenes
from lighter_gb300.scene import bake

pytestmark = pytest.mark.gpu
f32 = np.float32
SMALL = f32(0.001)


def dot(a, b):
    return a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1] + a[..., 2] * b[..., 2]


def brute(tri, seg):
    p1, p2, p3 = tri[:, 0:3], tri[:, 3:6], tri[:, 6:9]
    u, v = p2 - p1, p3 - p1
    n = np.stack([u[:, 1] * v[:, 2] - u[:, 2] * v[:, 1], u[:, 2] * v[:, 0] - u[:, 0] * v[:, 2],
                  u[:, 0] * v[:, 1] - u[:, 1] * v[:, 0]], 1)
    flat = (np.abs(n) < SMALL).all(1)
    uu, uv, vv = dot(u, u), dot(u, v), dot(v, v)
    D = uv * uv - uu * vv
    out = np.full(len(seg), 2.0, f32)
    with np.errstate(all="ignore"):
        for k, (a, b) in enumerate(zip(seg[:, :3], seg[:, 3:])):
            d = b - a
            nn, b_ = -dot(n, a - p1), dot(n, d[None])
            r = nn / b_
            w = (a + r[:, None] * d) - p1
            wu, wv = dot(w, u), dot(w, v)
            s, t = (uv * wv - vv * wu) / D, (uv * wu - uu * wv) / D
            ok = ~flat & ~(np.abs(b_) < SMALL) & ~(r < 0) & ~(r > 1) & ~(s < 0) & ~(s > 1) & ~(t < 0) & ~(s + t > 1)
            if ok.any():
                out[k] = r[ok].min()
    return out


def soup(n, seed, size=0.3):
    rng = np.random.default_rng([n, seed])
    c = rng.uniform(-5, 5, (n, 1, 3))
    return (c + rng.uniform(-size, size, (n, 3, 3))).astype(f32).reshape(n, 9)


def segments(m, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-6, 6, (m, 6)).astype(f32)


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 33, 1023, 1024, 1025, 1040, 2049, 8191, 8193, 20000])
def test_closest_hits_match_brute_force(gpu, n):
    tri, seg = soup(n, 1), segments(300, n)
    assert np.array_equal(ext.trace_segments(gpu, tri, seg), brute(tri, seg))


@pytest.mark.parametrize("n", [5, 1024, 1500, 9000])
def test_runs_of_equal_boxes(gpu, n):
    tri = np.repeat(soup(3, 7, 2.0), (n + 2) // 3, 0)[:n]
    seg = segments(200, 3)
    assert np.array_equal(ext.trace_segments(gpu, tri, seg), brute(tri[:: max(1, (n + 2) // 3)], seg))


@pytest.mark.parametrize("boxes,spheres", [(0, 1), (40, 4), (200, 40)])
def test_tree_reaches_every_leaf_once(gpu, monkeypatch, boxes, spheres):
    monkeypatch.setenv("LTRG_VALIDATE", "1")   # the bake re-checks the topology after the build
    bake(gpu, scenes.mid(3, lm=64, n_boxes=boxes, n_spheres=spheres, bounces=0, ao_rays=4), debug=False)


def test_unordered_boxes_are_an_error(gpu):
    tri = soup(50, 2)
    tri[7, 3] = np.inf
    with pytest.raises(RuntimeError):
        ext.trace_segments(gpu, tri, segments(5, 1))
    tri = soup(3000, 2)
    tri[1500, 3] = np.inf
    with pytest.raises(RuntimeError):
        ext.trace_segments(gpu, tri, segments(5, 1))
    assert np.array_equal(ext.trace_segments(gpu, tri[:1500], segments(9, 1)), brute(tri[:1500], segments(9, 1)))
