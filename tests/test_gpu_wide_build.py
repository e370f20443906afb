"""The four-wide form of hierarchies whose leaves have every size (needs a B200).

Coincident spheres make leaves of any size (a node whose centroids coincide is never split). The
form places records in leaf pairs by a scan in chunks of 1,024 records, so leaves start, end and
continue on either side of chunk edges here. Hits must equal the oracle's, and images through the
form those through the pairs.
"""

import numpy as np
import pytest

import oracle
from test_gpu_wide import assert_same_image, scene_of
from toaster_b200 import configs
from toaster_b200.scene import scene_to_gpu

pytestmark = pytest.mark.gpu


def clustered(sizes, seed):
    """Groups of coincident spheres of different radii, one group per entry of `sizes`, and a few
    triangles."""
    rng = np.random.default_rng(seed)
    scene = scene_of(5, 1, seed)
    centers = rng.uniform(-1.0, 1.0, (len(sizes), 3)).astype(np.float32)
    scene.sphere_centers = np.repeat(centers, sizes, axis=0)
    n = len(scene.sphere_centers)
    scene.sphere_radii = rng.uniform(0.02, 0.3, n).astype(np.float32)
    scene.sphere_materials = (np.arange(n) % 3).astype(np.uint32)
    return scene


SIZES = [[5], [1018], [1019], [1020], [2500], [999, 7, 1025, 2, 64, 3000, 1], [8] * 300]


@pytest.mark.parametrize("sizes", SIZES, ids=[f"{len(s)}x{max(s)}" for s in SIZES])
def test_leaves_of_every_size(renderer, sizes):
    scene, moved = clustered(sizes, 5), clustered(sizes, 6)
    rays = configs.parity_rays(scene, 5001, seed=1)
    renderer.upload(scene_to_gpu(scene))
    prim, t = renderer.trace_closest(rays)
    want_prim, want_t = oracle.Oracle(scene).trace_closest(rays)
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))
    assert_same_image(renderer)
    renderer.update_geometry(scene_to_gpu(moved))
    assert_same_image(renderer)


# The automatic choice of the builder remembers a degenerate leaf below 4,096 primitives: whatever came
# before, each scene gets the hierarchy of a host build.
def test_build_choice_after_a_degenerate_leaf(renderer):
    regular, degenerate = scene_of(1500, 20, 2), scene_of(1500, 20, 2, coincident=True)
    rays = configs.parity_rays(regular, 5001, seed=2)

    def hits(scene, mode):
        renderer.set_hierarchy_build(mode)
        try:
            renderer.upload(scene_to_gpu(scene))
        finally:
            renderer.set_hierarchy_build("auto")
        return renderer.stats()["bvh_depth"], renderer.trace_closest(rays)

    want = {id(s): hits(s, "host") for s in (degenerate, regular)}
    for scene in (degenerate, degenerate, regular, regular, degenerate):
        depth, (prim, t) = hits(scene, "auto")
        want_depth, (want_prim, want_t) = want[id(scene)]
        assert depth == want_depth
        assert np.array_equal(prim, want_prim) and np.array_equal(t.view(np.uint32), want_t.view(np.uint32))
