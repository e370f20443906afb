"""Rays and hierarchies at the edges of what the four-wide traversal takes (needs a B200).

Closest hits through the four-wide form against the oracle, or bit for bit against the pair traversal
on the device: a hierarchy whose root box is larger than need be has no four-wide form and the same
order of visits.
"""

import numpy as np
import pytest

import oracle
from test_gpu_animation_hierarchy import own_tree
from test_gpu_wide import assert_same_image, scene_of
from toaster_b200 import configs, gpu_types as gt, native
from toaster_b200.scene import scene_to_gpu

pytestmark = pytest.mark.gpu


def lattice():
    """Touching spheres of radius 1/2 on integer points, each twice: box faces that rays start on and
    exact ties."""
    scene = scene_of(0, 1, 1)
    g = np.stack(np.meshgrid(*[np.arange(-2, 3)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    scene.sphere_centers = np.concatenate([g, g[::-1]])
    n = len(scene.sphere_centers)
    scene.sphere_radii = np.full(n, 0.5, np.float32)
    scene.sphere_materials = (np.arange(n) % 3).astype(np.uint32)
    return scene


@pytest.mark.parametrize("tmin", [0.0, 0.001])
def test_axis_parallel_rays_from_box_faces(renderer, tmin):
    rng = np.random.default_rng(3)
    n = 60000
    rays = np.zeros((n, 6), np.float32)
    rays[:, :3] = rng.integers(-6, 7, (n, 3)) * np.float32(0.5)
    rays[:, 3:] = rng.choice(np.array([0.0, -0.0, 0.0, 1.0, -1.0, 0.5], np.float32), (n, 3))
    rays[:, 3:][np.all(rays[:, 3:] == 0, axis=1), 1] = 1.0
    scene = lattice()
    renderer.upload(scene_to_gpu(scene))
    prim, t = renderer.trace_closest(rays, tmin)
    want_prim, want_t = oracle.Oracle(scene).trace_closest(rays, tmin)
    assert np.mean(prim != 0xFFFFFFFF) > 0.2
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))


@pytest.mark.parametrize("scene", [scene_of(700, 20, 5), lattice()], ids=["random", "lattice"])
@pytest.mark.parametrize("tmin", [0.001, 0.0, 1.0])
def test_extreme_rays_hit_what_the_pairs_hit(renderer, scene, tmin):
    rng = np.random.default_rng(8)
    n = 40000
    rays = configs.parity_rays(scene, n, seed=2)
    values = np.array([0.0, -0.0, 1.0, -0.5, 1e-45, -1e-40, 1e-38, 1e-20, 1e15, -1e25, 3e38, np.inf, -np.inf, np.nan],
                      np.float32)
    for axis in range(6):
        pick = rng.random(n) < (0.1 if axis < 3 else 0.3)
        rays[pick, axis] = rng.choice(values, int(pick.sum()))
    d = scene_to_gpu(scene)
    nodes, refs = native.build_bvh_host(d.spheres, d.triangles)
    hits = []
    for loosen in (False, True):
        if loosen:
            nodes["max"][0, :3] += np.float32(0.25)
        renderer.upload(scene_to_gpu(scene, bvh=(nodes, refs)))
        hits.append(renderer.trace_closest(rays, tmin))
    (prim, t), (want_prim, want_t) = hits
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t, want_t, equal_nan=True)


def chain(n):
    """n overlapping spheres along the view, one leaf each, in a hierarchy of n levels."""
    scene = scene_of(0, 1, 1)
    scene.sphere_centers = np.stack([np.linspace(-0.3, 0.3, n), np.zeros(n), np.linspace(0.4, -0.4, n)], 1).astype("f4")
    scene.sphere_radii = np.linspace(0.2, 0.9, n).astype(np.float32)
    scene.sphere_materials = (np.arange(n) % 3).astype(np.uint32)
    return scene


def chained(scene, left):
    d = scene_to_gpu(scene)
    c, rad = d.spheres["center_radius"][:, :3], d.spheres["center_radius"][:, 3:]
    lo, hi, n = c - rad, c + rad, len(c)
    refs = np.zeros(n, gt.PRIMITIVE_REF)
    refs["index"] = np.arange(n)
    nodes = []

    def add(a, b):
        node = np.zeros(1, gt.BVH_NODE)
        node["min"][0, :3], node["max"][0, :3] = lo[a:b].min(axis=0), hi[a:b].max(axis=0)
        nodes.append(node)
        if b - a == 1:
            node["first_or_right"], node["primitive_count"] = a, 1
            return
        cut = b - 1 if left else a + 1
        add(a, cut)
        node["first_or_right"] = len(nodes)
        add(cut, b)

    add(0, n)
    return scene_to_gpu(scene, bvh=(np.concatenate(nodes), refs))


# 42 levels are the most the four-wide traversal's stack takes, 64 the pairs'.
@pytest.mark.parametrize("levels", [41, 42, 43, 64])
@pytest.mark.parametrize("left", [False, True])
def test_deep_hierarchies(renderer, levels, left):
    scene = chain(levels)
    renderer.upload(chained(scene, left))
    assert renderer.stats()["bvh_depth"] == levels
    rays = configs.parity_rays(scene, 20001, seed=6)
    prim, t = renderer.trace_closest(rays)
    want_prim, want_t = oracle.Oracle(scene).trace_closest(rays)
    assert np.array_equal(prim, want_prim)
    assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))
    assert_same_image(renderer)


@pytest.mark.parametrize("loosened", [False, True])
def test_order_of_a_loosened_box(renderer, loosened):
    """Two equal triangles of different materials in two subtrees: the one visited last is seen. A box
    made larger towards the camera is visited first, which its children's planes do not show."""
    scene = scene_of(4, 0, 1)
    big = np.array([[-3, -3, 0], [3, -3, 0], [0, 4, 0]], np.float32)
    small = np.array([[0, 0, -0.5], [0.1, 0, -0.5], [0, 0.1, -0.5]], np.float32)
    scene.triangles = np.stack([big, small, big, small])
    scene.triangle_materials = np.array([0, 2, 1, 2], np.uint32)
    data = own_tree(scene, 1)
    refs = data.bvh_primitives
    refs["kind"], refs["index"] = 1, np.arange(4)
    nodes = data.bvh_nodes
    assert list(nodes["primitive_count"]) == [0, 0, 1, 1, 0, 1, 1]
    lo, hi = scene.triangles.min(axis=1) - np.float32(1e-5), scene.triangles.max(axis=1) + np.float32(1e-5)
    for k, prims in enumerate([[0, 1, 2, 3], [0, 1], [0], [1], [2, 3], [2], [3]]):
        nodes["min"][k, :3], nodes["max"][k, :3] = lo[prims].min(axis=0), hi[prims].max(axis=0)
    if loosened:
        nodes["max"][1, 2] += np.float32(1.0)
    renderer.upload(data)
    rays = configs.parity_rays(scene, 2000, seed=1)
    prim, _ = renderer.trace_closest(rays)
    seen = prim[(prim & 0x7FFFFFFF) % 2 == 0]
    front = prim[:1000][(prim[:1000] != 0xFFFFFFFF) & ((prim[:1000] & 0x7FFFFFFF) % 2 == 0)]
    assert len(front) > 100 and len(seen) >= len(front)
    assert np.all((front & 0x7FFFFFFF) == (2 if loosened else 0))
    assert_same_image(renderer)
