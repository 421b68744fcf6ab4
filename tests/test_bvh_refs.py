"""Leaf references of long triangles (split at midpoints of their box) beside triangles that keep their own box: closest
hits through the tree against the segment test over every triangle, which do not depend on the references as long as no
piece is missing. Lattice triangles put vertices and whole edges on the cut planes; `scale` moves extents from
within the limit (four median extents) across it."""
import numpy as np
import pytest

from lighter_gb300 import ext
from test_bvh_build import brute, segments, soup

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("n_small,n_long", [(0, 1), (0, 3), (3, 2), (64, 1), (63, 40), (500, 200)])
@pytest.mark.parametrize("scale", [1.0, 2.5, 40.0])
def test_hits_with_split_triangles(gpu, n_small, n_long, scale):
    rng = np.random.default_rng([n_small, n_long])
    lattice = rng.integers(-2, 3, (n_long, 3, 3)).astype(f32) * f32(scale * 0.25)
    lattice[::2, :, rng.integers(0, 3)] = f32(scale * 0.125)   # axis-aligned: flat boxes
    tri = np.concatenate([soup(n_small, 5) if n_small else np.zeros((0, 9), f32), lattice.reshape(-1, 9)])
    tri = tri[rng.permutation(len(tri))]
    seg = segments(300, n_long)
    assert np.array_equal(ext.trace_segments(gpu, tri, seg), brute(tri, seg))
