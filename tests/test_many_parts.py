"""A mesh cut into thousands of parts bakes to the bits of the same triangles in one part, and in about its time: what
the host prepares per part must not grow with the parts before it (copying the triangles so far for each of 8,192 parts
took twenty times the bake)."""
import time

import numpy as np
import pytest

from lighter_gb300 import abi
from lighter_gb300.scene import Instance, Light, Mesh, Part, SceneDesc, ingest

pytestmark = pytest.mark.gpu
SIDE = 362   # 131,044 quads


def grid(parts):
    n = SIDE * SIDE
    k = np.arange(n)
    corner = np.array([[0, 0], [0.9, 0], [0.9, 0.9], [0, 0.9]])
    xy = np.stack([k % SIDE, k // SIDE], 1)[:, None] + corner
    uv = (np.stack([k % SIDE, k // SIDE], 1)[:, None] + 0.05 + corner) / SIDE
    pos = np.concatenate([xy * 20.0 / SIDE, np.zeros((n, 4, 1))], 2).astype(np.float32)
    cuts = np.linspace(0, n, parts + 1).astype(int)
    out = []
    for a, b in zip(cuts[:-1], cuts[1:]):
        q = b - a
        idx = (4 * np.arange(q)[:, None] + np.array([0, 1, 2, 2, 3, 0])).ravel()
        t = uv[a:b].reshape(-1, 2).astype(np.float32)
        out.append(Part(pos[a:b].reshape(-1, 3), np.tile(np.array([0, 0, 1], np.float32), (4 * q, 1)), t, t,
                        idx.astype(np.uint32), 1))
    return SceneDesc("grid", [Mesh("grid", out)], [Instance(0)],
                     [Light(abi.LTR_LT_POINT, (5.0, 5.0, 5.0), range=60.0, shadow_sample_count=1)],
                     {"ao_distance": 0.0, "bounce_count": 0}, fixed_lm_size=(256, 256))


def test_time_does_not_follow_the_parts(gpu):
    ms, maps = [], []
    for parts in (1, 8192):
        scene, keep = ingest(gpu, grid(parts))
        try:
            best = 1e9
            for _ in range(3):
                t0 = time.perf_counter()
                gpu.ltr_Start(scene)
                assert gpu.ltrg_Wait(scene)
                best = min(best, time.perf_counter() - t0)
            ms.append(best * 1e3)
            wo = abi.WorkOutput()
            assert gpu.ltr_GetWorkOutput(scene, 0, wo)
            maps.append(np.ctypeslib.as_array(wo.lightmap_rgb, (256, 256, 3)).copy())
        finally:
            gpu.ltr_DestroyScene(scene)
    assert np.array_equal(*maps) and maps[0].any()
    assert ms[1] < 5 * ms[0], ms
