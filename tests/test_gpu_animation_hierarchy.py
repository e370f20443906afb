"""The scene a context holds around animations with a per-frame hierarchy build (needs a B200).

Such an animation puts its own median-split hierarchy in the place of the uploaded one, whatever
shape that had. Closest hits (oracle) and wavefront images (four-wide form against the pairs) show
which hierarchy the context is left with.
"""

import numpy as np
import pytest

import oracle
from test_gpu_wide import assert_same_image, scene_of
from toaster_b200 import configs, native
from toaster_b200.native import TcError
from toaster_b200.renderer import Animation, GpuRenderer
from toaster_b200.scene import scene_to_gpu

pytestmark = pytest.mark.gpu


def given(scene, loosened):
    """The scene with a hierarchy of its own; `loosened`: one interior box larger than it need be, so
    that the hierarchy has no four-wide form."""
    d = scene_to_gpu(scene)
    nodes, refs = native.build_bvh_host(d.spheres, d.triangles)
    if loosened:
        nodes["max"][np.nonzero(nodes["primitive_count"] == 0)[0][1], :3] += np.float32(0.25)
    return scene_to_gpu(scene, bvh=(nodes, refs))


def assert_hits(renderer, scene):
    rays = configs.parity_rays(scene, 20001, seed=4)
    prim, t = renderer.trace_closest(rays)
    want_prim, want_t = oracle.Oracle(scene).trace_closest(rays)
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))


@pytest.mark.parametrize("loosened", [False, True])
@pytest.mark.parametrize("why", ["count", "vertex", "guide"])
def test_refused_animation_leaves_the_scene(native_lib, loosened, why):
    scene, moved = scene_of(300, 10, 3), scene_of(300, 10, 4)
    first = scene_to_gpu(moved)
    if why == "count":
        first = scene_to_gpu(scene_of(299, 10, 4))
    elif why == "vertex":
        first.triangles["v1"][7, 1] = np.nan
    with GpuRenderer(0) as r:
        r.upload(given(scene, loosened))
        with pytest.raises(TcError):
            Animation(r, first, rebuild=True, guiding=why == "guide")
        assert_hits(r, scene)
        assert_same_image(r)
