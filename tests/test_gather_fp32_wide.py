"""The FP32 gather with few patches and very many right-hand sides (more than 65,535 groups of 32), against FP64 sweeps
over its form factors: every term is non-negative, so an FP32 sum of n products and its handful of partial sums is
off by at most (n + 16) units of 2^-24, relative to the entry, per bounce."""
import os
import subprocess
import sys

import numpy as np
import pytest

from lighter_gb300.gather import FP32, REFINE_NONE, Gather

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


SCRATCH = r"""
import numpy as np
import torch
from lighter_gb300 import library
from lighter_gb300.gather import FP32, REFINE_NONE, Gather
n, R = 500, 500_000
gen = torch.Generator(device="cuda").manual_seed(1)
rng = np.random.default_rng(2)
u = rng.normal(size=(n, 3))
u /= np.linalg.norm(u, axis=1, keepdims=True)
alb = torch.rand(n, 3, device="cuda", generator=gen) * 0.5 + 0.3
E = torch.rand(n, R, device="cuda", generator=gen) + 0.5
out = torch.empty_like(E)
with Gather(library(), np.zeros((0, 9), np.float32), (2 * u).astype(np.float32), -u, np.full(n, 2.0 / n, np.float32)) as g:
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g.solve_device(alb.data_ptr(), E.data_ptr(), R, 1, out.data_ptr(), FP32, REFINE_NONE)
    used = free - torch.cuda.mem_get_info()[0]
    assert used <= 2 * E.numel() * 4, used
    G = torch.from_numpy(g.G().astype(np.float64)).cuda()
    for c in (0, 96 * 1000, 96 * 3000, R - 1000):
        e = E[:, c:c + 1000].double()
        x = e * alb.double()[:, torch.arange(c, c + e.shape[1], device="cuda") % 3]
        want = e + G @ x
        assert bool(((out[:, c:c + 1000].double() - want).abs() <= (n + 16) * 2.0 ** -24 * want).all())
print("bounded")
"""


def test_scratch_stays_below_the_right_hand_sides(gpu):
    """A solve's own buffers, beside the caller's arrays, take no more than two such arrays (the sweeps' vectors); in a
    process of its own, whose memory pool holds nothing yet."""
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", SCRATCH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "bounded", r.stderr[-2000:]
