"""cudaDeviceReset between calls: what the library remembers of a device must not be a part of the context that the
reset ended. In a process of its own (the reset ends only that process's context)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes
import numpy as np
from lighter_gb300 import ext, library, scenes
from lighter_gb300.gather import Gather
from lighter_gb300.scene import bake
gpu = library()
rng = np.random.default_rng(0)
tri = (rng.uniform(-5, 5, (20000, 1, 3)) + rng.uniform(-0.3, 0.3, (20000, 3, 3))).astype(np.float32).reshape(-1, 9)
seg = rng.uniform(-6, 6, (200, 6)).astype(np.float32)

def work():
    out = [ext.trace_segments(gpu, tri, seg)]
    d = scenes.mid(2, lm=96, n_boxes=60, n_spheres=10, bounces=0, ao_rays=4)   # more than 8,192 references too
    d.config["blur_size"] = 5.0
    out += [x[3] for x in bake(gpu, d, debug=False).lightmaps]
    with Gather(gpu, tri[:50], seg[:, :3], seg[:, 3:], np.full(200, 0.1, np.float32)) as g:
        out.append(g.G())
        out.append(g.solve(np.full((200, 3), 0.5, np.float32), np.ones((200, 6), np.float32), 2)[0])
    return out

before = work()
HOW
after = work()
assert len(before) == len(after) and all(np.array_equal(a, b) for a, b in zip(before, after))
print("equal")
"""
HOW = {"driver": """
cuda = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuDevicePrimaryCtxReset_v2(dev) == 0
""", "runtime": """
import glob
names = glob.glob("/usr/local/cuda/lib64/libcudart.so*")
cudart = ctypes.CDLL(sorted(names)[0])
assert cudart.cudaSetDevice(0) == 0
assert cudart.cudaDeviceReset() == 0
"""}


@pytest.mark.parametrize("how", ["driver", "runtime"])
def test_bakes_and_gathers_after_a_reset(gpu, how):
    r = subprocess.run([sys.executable, "-c", CHILD.replace("HOW", HOW[how])], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "equal", r.stderr[-2000:]
