"""The caller's size_fn runs for several instances at a time, however small they are (the reference calls it from its
pool threads, lighter.cpp:292-341), once per instance and with its error ending nothing else."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from lighter_gb300 import abi
from lighter_gb300.scene import Instance, Light, Mesh, SceneDesc, bake
from lighter_gb300.scenes import _quad_part

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 16, 40])
def test_size_fn_runs_side_by_side(gpu, n):
    lock = threading.Lock()
    seen = {"now": 0, "most": 0, "names": []}

    def size(cfg, mi, mi_size, ii, ii_size, area, importance, out):
        with lock:
            seen["now"] += 1
            seen["most"] = max(seen["most"], seen["now"])
            seen["names"].append(C.string_at(ii, ii_size))
        time.sleep(0.02)
        with lock:
            seen["now"] -= 1
        out[0], out[1] = 16, 8
        return 1

    cb = abi.SIZE_FN(size)
    insts = []
    for i in range(n):
        m = np.eye(4, dtype=np.float32)
        m[3, 0] = 3 * i
        insts.append(Instance(0, m, ident=f"i{i}"))
    res = bake(gpu, SceneDesc("slow", [Mesh("quad", [_quad_part()])], insts,
                              [Light(abi.LTR_LT_POINT, (0.0, 0.0, 3.0), range=9.0, shadow_sample_count=1)],
                              {"ao_distance": 0.0, "bounce_count": 0, "size_fn": C.cast(cb, C.c_void_p).value}),
               debug=False)
    assert len(res.lightmaps) == n and all(x[3].shape == (8, 16, 3) for x in res.lightmaps)
    assert sorted(seen["names"]) == sorted(f"i{i}".encode() for i in range(n))
    assert seen["most"] >= min(n, 8), seen["most"]
