"""Gathers of several host threads whose solves run the same kernel with pipelines of different sizes: every solve
succeeds with the bits of the same solve alone."""
import threading

import numpy as np
import pytest

from lighter_gb300.gather import BF16, REFINE_NONE, REFINE_RHS, Gather

pytestmark = pytest.mark.gpu
N = 300


@pytest.mark.parametrize("refine", [REFINE_NONE, REFINE_RHS])
def test_threads_of_different_widths(gpu, refine):
    rng = np.random.default_rng(4)
    pos, nrm = rng.uniform(-3, 3, (N, 3)), rng.normal(size=(N, 3))
    albedo = rng.uniform(0.2, 0.8, (N, 3)).astype(np.float32)
    widths = (3, 45, 96, 160)
    E = [rng.uniform(0, 4, (N, R)).astype(np.float32) for R in widths]
    gathers = [Gather(gpu, np.zeros((0, 9), np.float32), pos, nrm, np.full(N, 0.05, np.float32)) for _ in widths]
    try:
        want = [g.solve(albedo, e, 2, BF16, refine)[0].copy() for g, e in zip(gathers, E)]
        bad = []
        start = threading.Barrier(len(widths))

        def work(k):
            start.wait()
            for _ in range(800):
                try:
                    if not np.array_equal(gathers[k].solve(albedo, E[k], 2, BF16, refine)[0], want[k]):
                        bad.append((widths[k], "bits"))
                except RuntimeError as e:
                    bad.append((widths[k], str(e)))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(widths))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, (len(bad), bad[0])
    finally:
        for g in gathers:
            g.close()
