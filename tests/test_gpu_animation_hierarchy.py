"""The scene a context holds around animations with a per-frame hierarchy build (needs a B200).

Such an animation puts its own median-split hierarchy in the place of the uploaded one, whatever
shape that had. Closest hits (oracle) and wavefront images (four-wide form against the pairs) show
which hierarchy the context is left with.
"""

import numpy as np
import pytest

import oracle
from test_gpu_wide import assert_same_image, scene_of
from toaster_b200 import configs, gpu_types as gt, native
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


def own_tree(scene, leaf):
    """The scene with a hierarchy that halves its primitives along x down to leaves of `leaf`."""
    d = scene_to_gpu(scene)
    c, rad = d.spheres["center_radius"][:, :3], d.spheres["center_radius"][:, 3:]
    v = np.stack([d.triangles[k][:, :3] for k in ("v0", "v1", "v2")]) if len(d.triangles) else np.zeros((3, 0, 3), "f4")
    pad = np.float32(1e-5)
    lo = np.concatenate([c - rad, v.min(axis=0) - pad])
    hi = np.concatenate([c + rad, v.max(axis=0) + pad])
    nodes, order = [], np.argsort(lo[:, 0], kind="stable")
    refs = np.zeros(len(order), gt.PRIMITIVE_REF)
    refs["kind"], refs["index"] = order >= len(c), np.where(order >= len(c), order - len(c), order)

    def add(a, b):
        node = np.zeros(1, gt.BVH_NODE)
        node["min"][0, :3], node["max"][0, :3] = lo[order[a:b]].min(axis=0), hi[order[a:b]].max(axis=0)
        nodes.append(node)
        if b - a <= leaf:
            node["first_or_right"], node["primitive_count"] = a, b - a
            return
        add(a, (a + b) // 2)
        node["first_or_right"] = len(nodes)
        add((a + b) // 2, b)

    add(0, len(order))
    return scene_to_gpu(scene, bvh=(np.concatenate(nodes), refs))


# Hierarchies of more (leaf 1) and of fewer pairs than the build that takes their place.
@pytest.mark.parametrize("leaf", [1, 40])
def test_update_after_a_rebuild_animation(native_lib, leaf):
    scenes = [scene_of(300, 10, k) for k in (3, 4, 5, 6)]
    with GpuRenderer(0) as r:
        r.upload(own_tree(scenes[0], leaf))
        assert_hits(r, scenes[0])
        with Animation(r, scene_to_gpu(scenes[1]), rebuild=True) as a:
            assert_hits(r, scenes[1])
            assert_same_image(r)
            a.frame(scene_to_gpu(scenes[2]), 1)
        assert_hits(r, scenes[2])
        r.update_geometry(scene_to_gpu(scenes[3]))
        assert_hits(r, scenes[3])
        assert_same_image(r)


def test_frames_of_a_replaced_hierarchy_are_refused(native_lib):
    first, moved = scene_of(300, 10, 3), scene_of(300, 10, 4)
    with GpuRenderer(0) as r:
        r.upload(own_tree(first, 1))
        with Animation(r, scene_to_gpu(first)) as refit, Animation(r, scene_to_gpu(first), rebuild=True) as rebuild:
            with pytest.raises(TcError, match="replaced the hierarchy"):
                refit.frame(scene_to_gpu(moved), 1)
            rebuild.frame(scene_to_gpu(moved), 1)
        assert_hits(r, moved)


# Spheres and triangles change places between the frames' leaf orders when the hierarchy is rebuilt.
@pytest.mark.parametrize("rebuild", [False, True])
@pytest.mark.parametrize("triangles,spheres", [(0, 3), (7, 2), (700, 60)])
def test_four_wide_form_follows_captured_frames(native_lib, triangles, spheres, rebuild):
    scenes = [scene_of(triangles, spheres, k) for k in (7, 8, 9)]
    with GpuRenderer(0) as r:
        r.upload(scene_to_gpu(scenes[0]))
        with Animation(r, scene_to_gpu(scenes[0]), rebuild=rebuild) as a:
            for k in (1, 2):
                a.frame(scene_to_gpu(scenes[k]), k)
                assert_hits(r, scenes[k])
                assert_same_image(r)


def test_refused_upload_leaves_the_scene(native_lib):
    scene, other = scene_of(300, 10, 3), scene_of(900, 30, 4)
    bad = given(other, False)
    leaf = np.nonzero(bad.bvh_nodes["primitive_count"])[0]
    bad.bvh_nodes["first_or_right"][leaf[3]] = bad.bvh_nodes["first_or_right"][leaf[2]]
    with GpuRenderer(0) as r:
        r.upload(scene_to_gpu(scene))
        with pytest.raises(TcError, match="overlap|in no leaf"):
            r.upload(bad)
        assert_hits(r, scene)
        assert_same_image(r)
