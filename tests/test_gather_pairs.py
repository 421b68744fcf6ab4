"""The tensor-core gather on pairs of CTAs (split right-hand sides, N > 160, at least 16 units per SM): an even and an
odd number of 256-row blocks, a last row block of one row, n off the 64-wide k blocks, R on both sides of the MMA
widths 192, 224 and 256, and a wait that runs out.

Reference: FP64 sweeps over the FP32 form factors (ltrg_GatherGetG) rounded to 16 bits under the solve's power-of-two
scale (the largest factor below 2^14), whose heads the products read. Every term is non-negative. X is held as head
and tail: FP16 2^-22 of itself (11 + 11 bits), BF16 2^-18; an FP32 sum of n + 16 terms that truncates adds
(n + 16) * 2^-23.
"""
import numpy as np
import pytest

from lighter_gb300.gather import BF16, FP16, REFINE_RHS, Gather

pytestmark = pytest.mark.gpu


def _sphere(n, seed):
    rng = np.random.default_rng([n, seed])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    pos = (u * rng.uniform(1.5, 2.5, (n, 1))).astype(np.float32)   # facing the centre: linked, no occluders
    return pos, -u, rng.uniform(1.0 / n, 8.0 / n, n).astype(np.float32), rng


def _round16(G, precision):
    exp = 14 - np.frexp(G.max())[1]
    s = np.ldexp(G.astype(np.float32), exp)
    if precision == FP16:
        h = s.astype(np.float16).astype(np.float64)
    else:
        b = s.view(np.uint32).astype(np.uint64)
        h = ((b + 0x7fff + ((b >> 16) & 1)) & 0xffff0000).astype(np.uint32).view(np.float32).astype(np.float64)
    return np.ldexp(h, -exp)


@pytest.mark.parametrize("n,R", [(6500, 161), (6500, 192), (6657, 193), (6701, 225), (7169, 256)])
@pytest.mark.parametrize("precision", [FP16, BF16])
def test_pairs_against_fp64(gpu, n, R, precision):
    pos, nrm, area, rng = _sphere(n, R)
    albedo = rng.uniform(0.3, 0.8, (n, 3)).astype(np.float32)
    E = rng.uniform(0.0, 5.0, (n, R)).astype(np.float32)
    bounces = 2
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, nrm, area) as g:
        G16 = _round16(g.G(), precision)
        B, st = g.solve(albedo, E, bounces, precision, REFINE_RHS)
        again, _ = g.solve(albedo, E, bounces, precision, REFINE_RHS)
    assert st["tensor_cores"] == 1 and st["ctas"] % 2 == 0 and st["stages"] > 2
    cols = rng.choice(R, 24, replace=False)
    cols[:2] = 0, R - 1
    alb = albedo.astype(np.float64)[:, cols % 3]
    want = E[:, cols].astype(np.float64)
    for _ in range(bounces):
        want = E[:, cols] + G16 @ (alb * want)
    rel = np.abs(B[:, cols] - want) / want
    assert rel.max() <= bounces * (2.0 ** (-22 if precision == FP16 else -18) + (n + 16) * 2.0 ** -23)
    assert np.array_equal(B, again)


@pytest.mark.parametrize("chunk", [1, 7, 64])
def test_pairs_in_chunks(gpu, chunk):
    """Accumulation in chunks of k blocks: more accumulator hand-overs between the pair's issuer and both epilogues."""
    n, R = 6657, 192
    pos, nrm, area, rng = _sphere(n, chunk)
    albedo = rng.uniform(0.3, 0.8, (n, 3)).astype(np.float32)
    E = rng.uniform(0.0, 5.0, (n, R)).astype(np.float32)
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, nrm, area) as g:
        G16 = _round16(g.G(), FP16)
        g.set_chunk(chunk)
        B, st = g.solve(albedo, E, 1, FP16, REFINE_RHS)
    assert st["ctas"] % 2 == 0 and st["stages"] > 2
    want = E + G16 @ (albedo.astype(np.float64)[:, np.arange(R) % 3] * E)
    assert (np.abs(B - want) / want).max() <= 2.0 ** -22 + (n + 16) * 2.0 ** -23


def test_pair_wait_expires_and_the_next_solve_succeeds(gpu):
    pos, nrm, area, rng = _sphere(6700, 0)
    albedo = np.full((6700, 3), 0.5, np.float32)
    E = rng.uniform(0.0, 5.0, (6700, 192)).astype(np.float32)
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, nrm, area) as g:
        ref, _ = g.solve(albedo, E, 2, FP16, REFINE_RHS)
        g.stall_next_solve(20000)
        kept = np.full_like(E, 7.0)
        with pytest.raises(RuntimeError, match="wait expired"):
            g.solve(albedo, E, 2, FP16, REFINE_RHS, out=kept)
        assert (kept == 7.0).all()
        again, _ = g.solve(albedo, E, 2, FP16, REFINE_RHS)
    np.testing.assert_array_equal(again, ref)
