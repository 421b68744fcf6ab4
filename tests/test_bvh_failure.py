"""A scene whose occluders cannot be ordered (an infinite vertex) ends its bake at the build: no later stage runs, so
the caller's sample_fn is never called; the next bake of the process is sound. Alone and in a batch beside a scene
that bakes."""
import numpy as np
import pytest

from lighter_gb300 import scenes
from lighter_gb300.scene import Instance, Mesh, bake, bake_batch

pytestmark = pytest.mark.gpu


def scene(calls, broken):
    d = scenes.cornell(6, lm=24, bounces=1, ao=True)
    d.sample_table = None

    def sample(req):
        calls.append(1)
        return False

    d.sample_fn_py = sample
    if broken:
        part = scenes.faces_to_part([np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]])], 24, 0)
        part.positions[1, 0] = np.inf
        d.meshes.append(Mesh("broken", [part]))
        d.instances.append(Instance(len(d.meshes) - 1, ident="broken"))
    return d


def test_bake_ends_at_the_build(gpu):
    calls = []
    with pytest.raises(RuntimeError, match="clustering"):
        bake(gpu, scene(calls, True), debug=False)
    assert not calls
    assert bake(gpu, scene(calls, False), debug=False).lightmaps and calls


def test_batch_scene_ends_at_the_build(gpu):
    calls, fine = [], []
    with pytest.raises(RuntimeError, match="scene 1 .*clustering"):
        bake_batch(gpu, [scene(fine, False), scene(calls, True)])
    assert not calls and fine
