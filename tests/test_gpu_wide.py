"""The four-wide traversal against the binary one (needs a B200).

Wavefront renders trace through the four-wide form of the hierarchy; with ``refill_lanes`` they
trace through the sibling pairs (the reference's node order, checked against the oracle elsewhere).
Both must find the same hits to the last bit, so at one sample per pixel, where every pixel's sum
is one path's radiance, the images must be equal exactly.
"""

import numpy as np
import pytest

import oracle
from toaster_b200 import configs, gpu_types as gt, native
from toaster_b200.scene import EnvironmentMap, Material, Scene, scene_to_gpu

pytestmark = pytest.mark.gpu


def scene_of(triangles: int, spheres: int, seed: int, coincident: bool = False) -> Scene:
    """Random triangles and spheres of every material kind in front of a camera, lit by a sky."""
    rng = np.random.default_rng(seed)
    mats = [Material.diffuse((0.6, 0.5, 0.7)), Material.metal((0.8, 0.8, 0.7), 0.1), Material.dielectric(1.5)]
    centers = rng.uniform(-1.0, 1.0, (spheres, 3)).astype(np.float32)
    if coincident:
        centers[:] = centers[0]
    tris = configs.random_triangles(triangles, seed, 0.1, 0.8) if triangles else np.zeros((0, 3, 3), np.float32)
    return Scene(
        camera_position=(0.0, 0.3, 3.5), camera_look_at=(0.0, 0.0, 0.0), fov_degrees=40.0, width=160, height=96,
        samples=1, max_bounces=6, background=gt.ENVIRONMENT, materials=mats,
        sphere_centers=centers, sphere_radii=rng.uniform(0.1, 0.5, spheres).astype(np.float32),
        sphere_materials=(np.arange(spheres) % 3).astype(np.uint32), triangles=tris,
        triangle_materials=(np.arange(triangles) % 3).astype(np.uint32),
        environment=EnvironmentMap(16, 8, rng.uniform(0.1, 1.0, (8, 16, 3)).astype(np.float32), 1.0, 0.0))


def sums(renderer, refill_lanes):
    renderer.render(samples=1, frame_index=5, schedule="wavefront", refill_lanes=refill_lanes)
    return renderer.readback_sums()[0], renderer.stats()["rays"]


def assert_same_image(renderer):
    wide, rays = sums(renderer, 0)
    pairs, pair_rays = sums(renderer, 2)
    assert rays == pair_rays
    assert np.array_equal(wide, pairs)
    assert wide.sum() > 0


# Leaves of one to four primitives and their remainders, one to many levels, one kind or both; many
# coincident spheres make one large leaf.
@pytest.mark.parametrize("triangles,spheres,coincident",
                         [(1, 0, False), (2, 0, False), (3, 0, False), (4, 0, False), (5, 0, False), (9, 0, False),
                          (0, 1, False), (0, 3, False), (0, 7, False), (3, 2, False), (1, 1, False), (67, 5, False),
                          (0, 33, True), (2, 9, True), (1025, 64, False), (6000, 3, False)])
def test_wide_traversal_finds_the_pairs_hits(renderer, triangles, spheres, coincident):
    renderer.upload(scene_to_gpu(scene_of(triangles, spheres, 100 + triangles + spheres, coincident)))
    assert_same_image(renderer)


def test_wide_form_follows_geometry_updates(renderer):
    first, moved = scene_of(700, 20, 1), scene_of(700, 20, 2)
    renderer.upload(scene_to_gpu(first))
    renderer.update_geometry(scene_to_gpu(moved))
    assert_same_image(renderer)


@pytest.mark.parametrize("loosened", [False, True])
def test_given_hierarchies(renderer, loosened):
    """A caller's own hierarchy; with an interior box larger than its children's union there is no
    wide form, and the pairs are traversed."""
    d = scene_to_gpu(scene_of(300, 10, 3))
    nodes, refs = native.build_bvh_host(d.spheres, d.triangles)
    if loosened:
        interior = np.nonzero(nodes["primitive_count"] == 0)[0]
        nodes["max"][interior[1], :3] += np.float32(0.25)
    renderer.upload(scene_to_gpu(scene_of(300, 10, 3), bvh=(nodes, refs)))
    assert_same_image(renderer)


# Ray counts around every change of the launch: one lane per warp, each power of two up to full
# warps, partial last pieces, more rays than one resident wave holds lanes.
@pytest.mark.parametrize("count", [1, 3, 31, 33, 127, 2368, 2369, 4737, 9473, 18945, 37889, 75777, 200003, 400001])
def test_hits_at_every_launch_shape(renderer, count):
    scene = scene_of(1500, 40, 9)
    rays = configs.parity_rays(scene, count, seed=count)
    rays[::7, 4] = 0.0  # axis-parallel components go to the pair traversal
    rays[::11, 3] = -0.0
    renderer.upload(scene_to_gpu(scene))
    prim, t = renderer.trace_closest(rays)
    want_prim, want_t = oracle.Oracle(scene).trace_closest(rays)
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t.view(np.uint32)[prim != 0xFFFFFFFF], want_t.view(np.uint32)[prim != 0xFFFFFFFF])


# Around the size from which uploads build on the device: the automatic choice, the host build and the
# device build must hold the same hierarchy, coincident centroids (a large leaf) included.
@pytest.mark.parametrize("triangles,spheres,coincident",
                         [(1020, 3, False), (1021, 3, False), (1022, 3, False), (2000, 60, False), (4090, 5, False),
                          (1100, 40, True)])
def test_builds_agree_around_the_device_threshold(renderer, triangles, spheres, coincident):
    scene = scene_of(triangles, spheres, 17, coincident)
    rays = configs.parity_rays(scene, 20001, seed=3)
    data, hits = scene_to_gpu(scene), {}
    for mode in ("host", "device", "auto"):
        renderer.set_hierarchy_build(mode)
        try:
            renderer.upload(data)
        finally:
            renderer.set_hierarchy_build("auto")
        hits[mode] = renderer.trace_closest(rays)
    for mode in ("device", "auto"):
        assert np.array_equal(hits[mode][0], hits["host"][0])
        assert np.array_equal(hits[mode][1].view(np.uint32), hits["host"][1].view(np.uint32))
