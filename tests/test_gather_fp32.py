"""The FP32 gather (k_sgemm_bounce, k_combine32) at the edges of its tiles: n around its 128-row tiles, k blocks of
32 and 4-float rows, R around each of its column tiles.

Reference: the same sweeps in FP64 over the FP32 form factors (ltrg_GatherGetG). Every term is non-negative, so an
FP32 sum of n products and its handful of partial sums is off by at most (n + 16) units of 2^-24, relative to
the entry, per bounce (the sum of n terms, the slots, the products with albedo, the emission).
"""
import numpy as np
import pytest

from lighter_gb300.gather import FP32, REFINE_NONE, Gather

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 31, 64, 127, 128, 129, 301, 1026])
@pytest.mark.parametrize("R", [1, 32, 33, 64, 95, 97, 192, 290])
def test_fp32_solve_tile_edges(gpu, n, R):
    rng = np.random.default_rng([n, R])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    pos = (u * rng.uniform(1.5, 2.5, (n, 1))).astype(np.float32)   # facing the centre: linked, no occluders
    area = rng.uniform(1.0 / n, 8.0 / n, n).astype(np.float32)
    albedo = rng.uniform(0.3, 0.8, (n, 3)).astype(np.float32)
    E = rng.uniform(0.0, 5.0, (n, R)).astype(np.float32)
    bounces = 2
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, -u, area) as g:
        G = g.G().astype(np.float64)
        B, st = g.solve(albedo, E, bounces, FP32, REFINE_NONE)
        again, _ = g.solve(albedo, E, bounces, FP32, REFINE_NONE)
    alb = albedo.astype(np.float64)[:, np.arange(R) % 3]
    want = E.astype(np.float64)
    for _ in range(bounces):
        want = E + G @ (alb * want)
    assert (G > 0).sum() > n * n // 2 - n
    rel = np.abs(B - want) / want
    assert rel.max() <= bounces * (n + 16) * 2.0 ** -24
    assert np.array_equal(B, again)
    assert st["tensor_cores"] == 0
