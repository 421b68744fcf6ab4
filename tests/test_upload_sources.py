"""Host arrays that a bake, a batch or a gather copies from live until the copies are done: with the allocator
overwriting memory as it is freed (MALLOC_PERTURB_), a copy that reads late would bring other bytes. Outputs are the
same bits as without."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import hashlib
import numpy as np
from lighter_gb300 import library, scenes
from lighter_gb300.gather import Gather
from lighter_gb300.scene import bake, bake_batch
gpu = library()
h = hashlib.sha256()
d = scenes.cornell(3, lm=48, bounces=1, ao=True)
d.config["generate_normalmap_data"] = 1
e = scenes.mid(2, lm=96, n_boxes=30, n_spheres=6, bounces=1, ao_rays=4)
e.config["ds2x"] = 1
e.config["blur_size"] = 17.0
for k in range(3):
    for res in [bake(gpu, d, gpu_options={"radiosity_patches": 40}), bake(gpu, e, debug=False)] + list(bake_batch(gpu, [d, e])[0]):
        for x in res.lightmaps:
            h.update(x[3].tobytes())
            if x[4] is not None:
                h.update(x[4].tobytes())
rng = np.random.default_rng(1)
tri = (rng.uniform(-2, 2, (300, 1, 3)) + rng.uniform(-0.3, 0.3, (300, 3, 3))).astype(np.float32).reshape(-1, 9)
pos = rng.uniform(-3, 3, (200, 3)).astype(np.float32)
for k in range(3):
    with Gather(gpu, tri, pos, rng.normal(size=(200, 3)), np.full(200, 0.1, np.float32)) as g:
        h.update(g.G().tobytes())
print(h.hexdigest())
"""


def run(**env):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env={**os.environ, **env}, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip()


def test_sources_outlive_their_copies(gpu):
    assert run(MALLOC_PERTURB_="165") == run()
