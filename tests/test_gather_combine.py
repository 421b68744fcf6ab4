"""The tensor-core gather's slot sums (k_combine) and G preparation (k_scale_cols, k_g_to_16) at the edges: 7, 8, 9 and
17 slots per 256-row block around the four or eight that are loaded at a time, grids on both sides of one tile and of
eight tiles per SM (152), n off the 4-float rows and 64-wide k blocks, R around the 32-wide tiles, through both host
paths and device arrays.

Reference: the same sweeps in FP64 over the FP32 form factors (ltrg_GatherGetG). Every term is non-negative. BF16
heads carry 9 bits (half an ulp is 2^-9 of the value); with the tails a factor is off by 2^-18 of itself and the
dropped tail-by-tail product by 2^-18 of the term, so a term is off by 3 * 2^-18; an FP32 sum of n + 16 terms that
truncates adds (n + 16) * 2^-23.
"""
import numpy as np
import pytest

from lighter_gb300.gather import BF16, REFINE_FULL, Gather

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(n, R) for n in (3, 447, 509, 512, 514, 1030) for R in (1, 32, 33, 100)] +
                         [(1200, 100), (1280, 128), (6500, 161), (6501, 193)])
def test_slot_sums_at_the_edges(gpu, n, R):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng([n, R, 7])
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    pos = (u * rng.uniform(1.5, 2.5, (n, 1))).astype(np.float32)   # facing the centre: linked, no occluders
    area = rng.uniform(1.0 / n, 8.0 / n, n).astype(np.float32)
    albedo = rng.uniform(0.3, 0.8, (n, 3)).astype(np.float32)
    E = rng.uniform(0.0, 5.0, (n, R)).astype(np.float32)
    bounces = 2
    with Gather(gpu, np.zeros((0, 9), np.float32), pos, -u, area) as g:
        G = g.G().astype(np.float64)
        B, st = g.solve(albedo, E, bounces, BF16, REFINE_FULL)
        g.host_path(1)
        staged, _ = g.solve(albedo, E, bounces, BF16, REFINE_FULL)
        d = [torch.from_numpy(a).cuda() for a in (albedo, E)]
        out = torch.empty_like(d[1])
        torch.cuda.synchronize()
        g.solve_device(d[0].data_ptr(), d[1].data_ptr(), R, bounces, out.data_ptr(), BF16, REFINE_FULL)
    alb = albedo.astype(np.float64)[:, np.arange(R) % 3]
    want = E.astype(np.float64)
    for _ in range(bounces):
        want = E + G @ (alb * want)
    assert st["tensor_cores"] == 1 and np.isfinite(G).all()
    rel = np.abs(B - want) / want
    assert rel.max() <= bounces * (3 * 2.0 ** -18 + (n + 16) * 2.0 ** -23)
    assert np.array_equal(B, staged) and np.array_equal(B, out.cpu().numpy())
