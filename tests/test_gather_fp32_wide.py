"""The FP32 gather with few patches and very many right-hand sides (more than 65,535 groups of 32), against FP64 sweeps
over its form factors: every term is non-negative, so an FP32 sum of n products and its handful of partial sums is
off by at most (n + 16) units of 2^-24, relative to the entry, per bounce."""
import numpy as np
import pytest

from lighter_gb300.gather import FP32, REFINE_NONE, Gather

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(3, 2_097_121), (2, 2_500_000)])
def test_millions_of_right_hand_sides(gpu, n, R):
    rng = np.random.default_rng([n, R])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    pos = (2 * u).astype(np.float32)
    albedo = rng.uniform(0.3, 0.8, (n, 3)).astype(np.float32)
    E = rng.uniform(0.5, 5.0, (n, R)).astype(np.float32)
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, -u, np.full(n, 0.5, np.float32)) as g:
        G = g.G().astype(np.float64)
        B, _ = g.solve(albedo, E, 2, FP32, REFINE_NONE)
    assert (G > 0).any()
    alb = albedo.astype(np.float64)[:, np.arange(R) % 3]
    want = E.astype(np.float64)
    for _ in range(2):
        want = E + G @ (alb * want)
    assert (np.abs(B - want) <= 2 * (n + 16) * 2.0 ** -24 * want).all()
