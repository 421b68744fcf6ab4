"""The sample fixup's two ways (k_fix_quick, k_fixup): a scene with a sliver triangle far from everything else sends
every sample through the reference-shaped trees, the same scene with a well-shaped one only those that some triangle
can push. Positions and lightmaps of the scene proper must be equal bit for bit."""
import numpy as np
import pytest

from lighter_gb300 import scenes
from lighter_gb300.scene import Instance, Mesh, bake

pytestmark = pytest.mark.gpu


def with_far_triangle(d, height):
    far = [np.array([[500.0, 500, 500], [510, 500, 500], [505, 500 + height, 500]])]
    d.meshes.append(Mesh("far", [scenes.faces_to_part(far, 16, 0)]))
    d.instances.append(Instance(len(d.meshes) - 1, shadow=0, ident="far"))
    return d


@pytest.mark.parametrize("make", [
    lambda: scenes.cornell(4, lm=512, bounces=0, ao=False),
    lambda: scenes.mid(2, lm=900, n_boxes=80, n_spheres=50, bounces=0, ao_rays=0),
    lambda: scenes.large(3, lm=1100, grid=(64, 32), tiles=(2, 1), n_rocks=40, n_points=2, ao_rays=0, bounces=0),
])
@pytest.mark.parametrize("correct", [None, 0.0])
def test_listing_every_sample_changes_nothing(gpu, make, correct):
    res = []
    for height in (8.0, 0.01):   # 80% and 0.1% of the longest edge
        d = with_far_triangle(make(), height)
        d.lights = d.lights[:1]
        if correct is not None:
            d.config["max_correct_dist"] = correct
        res.append(bake(gpu, d))
    quick, slow = res
    assert sum(len(x["loc"]) for x in quick.debug) >= 1 << 20   # k_fix_quick's range
    for i in range(1, len(quick.debug) - 1):   # instance 0: probes; the last one: the far triangle
        assert np.array_equal(quick.debug[i]["pos"], slow.debug[i]["pos"])
        assert np.array_equal(quick.debug[i]["nrm"], slow.debug[i]["nrm"])
    for a, b in zip(quick.lightmaps[:-1], slow.lightmaps[:-1]):
        assert np.array_equal(a[3], b[3])
