"""Two branches of the BVH build that ordinary scenes do not take: 4-wide nodes (from 2^18 leaf references on; the any-hit
walk of form factors reads them) and the radix hierarchy in place of a clustering tree deeper than 40. Visibility does
not depend on triangles that no segment meets, so the form factors of a soup are the same bits with and without enough
far triangles to take the other branch; closest hits are compared with the segment test over every triangle."""
import numpy as np
import pytest

from lighter_gb300 import ext
from lighter_gb300.gather import Gather
from test_bvh_build import brute, soup

f32 = np.float32


def chain(n, centre, size):
    """n triangles, each 1.02 times the one before about the same centre: nested boxes, so the cheapest merge is always
    the whole chain so far with the next one, and the clustering's tree is n - 1 deep."""
    t = np.array([[-1, -1, -1], [1, -0.5, 0.2], [0.3, 1, 1]])
    s = size * 1.02 ** np.arange(n)
    return (np.asarray(centre) + s[:, None, None] * t).astype(f32).reshape(n, 9)


def clustering_depth(tri):
    """Depth of the clustering's tree over boxes in list order (k_ploc's rules: 16 neighbours either way, least merged
    area, then distance, parity and place of the lower position)."""
    p = tri.reshape(-1, 3, 3).astype(np.float64)
    cl = [(a, b, 0) for a, b in zip(p.min(1), p.max(1))]

    def cost(i, j):
        e = np.maximum(cl[i][1], cl[j][1]) - np.minimum(cl[i][0], cl[j][0])
        return e[0] * e[1] + e[1] * e[2] + e[2] * e[0], abs(i - j), min(i, j) & 1, min(i, j)

    while len(cl) > 1:
        near = [min((j for j in range(max(0, i - 16), min(len(cl), i + 17)) if j != i), key=lambda j, i=i: cost(i, j))
                for i in range(len(cl))]
        out = []
        for i, j in enumerate(near):
            if near[j] != i:
                out.append(cl[i])
            elif i < j:
                a, b = cl[i], cl[j]
                out.append((np.minimum(a[0], b[0]), np.maximum(a[1], b[1]), max(a[2], b[2]) + 1))
        cl = out
    return cl[0][2]


def test_the_chain_is_deep():
    assert clustering_depth(chain(90, (0, 0, 0), 0.05)) == 89
    assert clustering_depth(soup(90, 1)) < 40


@pytest.mark.gpu
@pytest.mark.parametrize("n", [30, 41, 42, 60, 90])
@pytest.mark.parametrize("others", [0, 700, 5000])
def test_hits_in_a_deep_tree(gpu, n, others):
    centre = np.array([20.0, 3.0, -2.0])
    tri = chain(n, centre, 0.1)
    if others:
        tri = np.concatenate([soup(others, 4), tri])
    rng = np.random.default_rng([n, others])
    a = centre + rng.normal(size=(300, 3)) * 0.8
    seg = np.concatenate([a, 2 * (centre + rng.normal(size=(300, 3)) * 0.1) - a], 1).astype(f32)
    want = brute(tri, seg)
    assert (want < 2).sum() > 50
    assert np.array_equal(ext.trace_segments(gpu, tri, seg), want)


def far_soup(n, seed):
    """Triangles outside the ball of radius 9 that holds every segment."""
    rng = np.random.default_rng([n, seed])
    u = rng.normal(size=(n, 1, 3))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    return (u * rng.uniform(9, 60, (n, 1, 1)) + rng.uniform(-0.06, 0.06, (n, 3, 3))).astype(f32).reshape(n, 9)


@pytest.mark.gpu
@pytest.mark.parametrize("links", [ext.LTRG_LINKS_REFERENCE, ext.LTRG_LINKS_VISIBLE])
def test_wide_nodes_see_what_the_binary_walk_sees(gpu, links):
    rng = np.random.default_rng(8)
    n = 220
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    inside = (rng.uniform(-4, 4, (30000, 1, 3)) + rng.uniform(-0.06, 0.06, (30000, 3, 3))).astype(f32).reshape(-1, 9)
    G = []
    for extra in (far_soup(150_000, 1), far_soup(260_000, 1),
                  np.concatenate([far_soup(260_000, 1), chain(60, (40.0, 40.0, 40.0), 0.03)])):
        tri = np.concatenate([inside, extra])
        with Gather(gpu, tri, (7 * u).astype(f32), -u, np.full(n, 0.3, f32), links=links) as g:
            G.append(g.G())
    off = ~np.eye(n, dtype=bool)
    assert 0.1 < (G[0][off] > 0).mean() < 0.9
    assert np.array_equal(G[0], G[1]) and np.array_equal(G[0], G[2])
