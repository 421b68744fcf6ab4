"""Probe samples in a scene whose lightmaps cover no texel: patch radiosity has no patches, and the probes get what they
get without bounces (a probe's own diffuse and emission are zero)."""
import numpy as np
import pytest

from lighter_gb300 import abi
from lighter_gb300.scene import Instance, Light, Mesh, SceneDesc, bake
from lighter_gb300.scenes import _quad_part

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [0, 2])
def test_patch_radiosity_with_probes_alone(gpu, instances):
    part = _quad_part()
    part.uv2 = part.uv2 - 5.0   # no texel is covered
    colors = []
    for bounces in (0, 1):
        d = SceneDesc("probes", [Mesh("quad", [part])], [Instance(0)] * instances,
                      [Light(abi.LTR_LT_POINT, (0.5, 0.2, 3.0), range=9.0, power=1.0, shadow_sample_count=1)],
                      {"ao_distance": 0.0, "bounce_count": bounces}, fixed_lm_size=(16, 16),
                      probes=[(k, (0.1 * k, 0.2, 1.0), (0.0, 0.0, 1.0)) for k in range(7)])
        res = bake(gpu, d, gpu_options={"radiosity_patches": 30})
        assert not any(x[3].any() for x in res.lightmaps)
        colors.append(res.sample_colors)
    assert colors[0].any() and np.array_equal(*colors)
