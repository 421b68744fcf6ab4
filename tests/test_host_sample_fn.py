"""Radiosity with a sample_fn of the caller's (called on the host, its colours copied to the device) against the same
colours from the library's table function (evaluated on the device): the same bits, sample by sample and in patches, with a
direct-light stage long enough that the copies are queued behind it, alone and in a batch."""
import numpy as np
import pytest

from lighter_gb300 import scenes
from lighter_gb300.scene import bake, bake_batch

pytestmark = pytest.mark.gpu


def pair(lm):
    """The room under the table function and under a Python function that reads the same table."""
    out = []
    for host in (False, True):
        d = scenes.cornell(9, lm=lm, bounces=2, ao=False)
        dif = np.asarray(d.sample_table[0], np.float32)
        emi = np.random.default_rng(2).uniform(0, 0.3, dif.shape).astype(np.float32)
        d.sample_table = (dif, emi)
        if host:
            def sample(req, dif=dif, emi=emi):
                k = int(req.tex0u)
                if k >= len(dif):
                    return False
                req.out_diffuse_color[:] = [float(v) for v in dif[k]]
                req.out_emissive_color[:] = [float(v) for v in emi[k]]
                return True
            d.sample_table, d.sample_fn_py = None, sample
        out.append(d)
    return out


@pytest.mark.parametrize("patches,lm", [(0, 12), (60, 12), (150, 40)])
def test_host_function_equals_table(gpu, patches, lm):
    table, host = pair(lm)
    opts = {"radiosity_patches": patches}
    a = bake(gpu, table, debug=False, gpu_options=opts)
    runs = [bake(gpu, host, debug=False, gpu_options=opts), *bake_batch(gpu, [host, host], gpu_options=opts)[0]]
    assert any(x[3].any() for x in a.lightmaps)
    for r in runs:
        for x, y in zip(a.lightmaps, r.lightmaps):
            assert np.array_equal(x[3], y[3])
