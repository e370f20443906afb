"""Workloads of this framework for timing, through its public entry points.

Each case is a dict of plain values; ``prepare`` makes what a program holds before the call (scene
uploaded to a context, network weights, ray buffers), ``run`` makes one pass and returns its whole
outputs. The kinds and the ranges they stand for:

  hits       closest-hit queries, 2^10 to 2^20 rays from host arrays (picking, visibility queries)
             or device buffers, against scenes of 2,000 to 2.1 M primitives
  frame      one plain frame: render and read back the linear-HDR image, from a 320x180 preview to
             1920x1080, 1 to 64 samples per pixel, 3 to 8 bounces; with moments the FP64 sums come back
  progressive  a plain image accumulated in several batches, FP64 sums read back
  guided     one guided frame, recording its training samples where it is large enough
  edit       a scene edit: upload the packed records, render a preview, read the display image back
  batch      several small scenes of uneven size in one call
  animation  one animated frame: geometry in, display image out (per-frame hierarchy build or refit)
  train      loss and weight gradient of the guiding network on a batch of samples

Scenes are the seeded generators of ``toaster_b200.configs``. Path tracing draws random numbers of
its own, so rendered images have no closed-form value: ``exact`` covers hit distances and gradients.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from toaster_b200 import configs, guiding_eval
from toaster_b200 import gpu_types as gt
from toaster_b200.renderer import Animation, GpuRenderer, render_batch
from toaster_b200.scene import scene_to_gpu


def listed() -> list:
    return [
        # The smallest call: a few thousand rays from a host array (smoke-test size).
        {"name": "hits_small", "kind": "hits", "scene": "small", "prims": 2048, "rays": 4096, "host": True,
         "watertight": False},
        # The parity ray set on the terrain of 2.1 M triangles, rays and hits in device memory.
        {"name": "hits_mesh", "kind": "hits", "scene": "mesh", "prims": 2093058, "rays": 1 << 20,
         "host": False, "watertight": False},
        # The small plain configuration, the size of the published fixture suite.
        {"name": "frame_small", "kind": "frame", "scene": "small", "prims": 2048, "width": 320, "height": 180,
         "spp": 4, "bounces": 4, "moments": False},
        # A window of odd size with error estimates (FP64 sums and sums of squares).
        {"name": "frame_odd", "kind": "frame", "scene": "mixed", "prims": 2048, "width": 417, "height": 235,
         "spp": 3, "bounces": 5, "moments": True},
        # The headline frame: mixed scene, 1280x720, 64 spp, 8 bounces.
        {"name": "frame_mixed", "kind": "frame", "scene": "mixed", "prims": 2048, "width": 1280, "height": 720,
         "spp": 64, "bounces": 8, "moments": False},
        # The large mesh at full HD, one progressive batch's worth of samples.
        {"name": "frame_mesh", "kind": "frame", "scene": "mesh", "prims": 2093058, "width": 1920, "height": 1080,
         "spp": 8, "bounces": 8, "moments": False},
        # The closed interior accumulated in batches (what an equal-time comparison's plain side does).
        {"name": "progressive_room", "kind": "progressive", "scene": "room", "prims": 8192, "width": 1280,
         "height": 720, "spp": 8, "batches": 2, "bounces": 8},
        # A guided batch of the same interior that records samples for online training.
        {"name": "guided_room", "kind": "guided", "scene": "room", "prims": 8192, "width": 1280, "height": 720,
         "spp": 4, "bounces": 8, "record": True},
        # An edited scene previewed: upload, 4 spp, display image.
        {"name": "edit_preview", "kind": "edit", "scene": "mixed", "prims": 2048, "width": 640, "height": 360,
         "spp": 4, "bounces": 8},
        # Thumbnails of several scenes in one call.
        {"name": "batch_previews", "kind": "batch", "scenes": 6, "min_width": 160, "max_width": 480, "spp": 4,
         "bounces": 4},
        # One frame of the ballistic animation with a per-frame hierarchy build.
        {"name": "animation", "kind": "animation", "width": 640, "height": 360, "spp": 16, "bounces": 8,
         "rebuild": True},
        # One training batch of the guiding network.
        {"name": "train_gradient", "kind": "train", "samples": 32768},
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _frame_size(rng, lo: int, hi: int) -> tuple:
    w = int(_log(rng, lo, hi))
    return w, max(16, int(w * rng.choice([9 / 16, 3 / 4, 0.41])))


def draw(rng) -> dict:
    kind = rng.choice(["hits", "hits", "frame", "frame", "frame", "progressive", "guided", "edit", "batch",
                       "animation", "train"])
    if kind == "hits":
        scene = rng.choice(["small", "mixed", "room", "mesh"])
        return {"kind": kind, "scene": scene, "prims": int(_log(rng, 500, 2e4 if scene != "mesh" else 1e6)),
                "rays": int(_log(rng, 1 << 10, 1 << 20)), "host": rng.random() < 0.4,
                "watertight": rng.random() < 0.15}
    if kind == "train":
        return {"kind": kind, "samples": int(_log(rng, 2048, 1 << 17))}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 8), "min_width": 160, "max_width": rng.choice([320, 480, 640]),
                "spp": rng.randint(1, 6), "bounces": rng.randint(3, 6)}
    scene = rng.choice(["small", "mixed", "room", "mesh"])
    case = {"kind": kind, "scene": scene, "prims": int(_log(rng, 500, 2e4 if scene != "mesh" else 1e6))}
    w, h = _frame_size(rng, 200, 1280)
    # Samples so that the call stays under 12 M paths (2 M for previews).
    most = 2e6 if kind == "edit" else 1.2e7
    spp = max(1, int(min(64, _log(rng, 1, 64), most / (w * h))))
    case.update(width=w, height=h, spp=spp, bounces=rng.randint(3, 8))
    if kind == "frame":
        case["moments"] = rng.random() < 0.3
    elif kind == "progressive":
        case["batches"] = rng.randint(2, 4)
        case["spp"] = max(1, spp // case["batches"])
    elif kind == "guided":
        case["scene"], case["spp"] = "room", max(1, min(spp, int(4e6 / (w * h))))
        case["record"] = w * h * case["spp"] >= 1 << 20  # smaller guided frames do not record
    elif kind == "animation":
        del case["scene"], case["prims"]
        case["rebuild"] = rng.random() < 0.5
        case["spp"] = max(1, spp // 2)
    return case


# ------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _sky():
    return configs.sky_environment()


def _scene(case: dict, seed: int):
    """A scene of about case["prims"] triangles with the case's frame settings."""
    kind, n = case["scene"], case["prims"]
    if kind == "small":
        s = configs.plain_small(seed)
        if n != 2048:
            s.triangles = np.concatenate([configs.random_triangles(n, seed), s.triangles[-2:]])
            s.triangle_materials = np.concatenate([np.arange(n) % 2048, [2049, 2049]]).astype(np.uint32)
    elif kind == "mixed":
        s = configs.mixed(seed, environment=_sky())
        if n != 2048:
            s.triangles = configs.random_triangles(n, seed)
            s.triangle_materials = (np.arange(n) % 2048).astype(np.uint32)
    elif kind == "room":
        s = configs.room_with_window(seed, clutter=n, environment=_sky())
    else:
        s = configs.large_mesh(seed, grid=max(8, int(round(math.sqrt(n / 2))) + 1), environment=_sky())
    if "width" in case:
        s.width, s.height, s.samples, s.max_bounces = case["width"], case["height"], case["spp"], case["bounces"]
    return s


def _pinned(*shape, dtype=torch.float32) -> np.ndarray:
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _training_samples(n: int, seed: int) -> np.ndarray:
    """(n, 10): surface points in a 4 x 3 x 4 room, unit normals, directions gathered around a window
    direction, weights with the long tail of recorded radiance."""
    rng = np.random.default_rng(seed)
    p = rng.uniform([-2.0, 0.0, -2.0], [2.0, 3.0, 2.0], (n, 3))
    unit = lambda v: v / np.linalg.norm(v, axis=1, keepdims=True)  # noqa: E731
    normal = unit(rng.normal(size=(n, 3)))
    window = unit(np.array([0.5, 1.8, 2.0]) - p + rng.normal(scale=0.3, size=(n, 3)))
    omega = np.where(rng.random((n, 1)) < 0.7, window, unit(rng.normal(size=(n, 3))))
    weight = np.minimum(rng.exponential(1.0, (n, 1)) ** 2, 50.0)
    return np.ascontiguousarray(np.concatenate([p, normal, omega, weight], axis=1), np.float32)


ROOM_BOUNDS = (0.0, 1.5, 0.0, 0.5)


def _batch_sizes(case: dict) -> list:
    """16:9 frames with widths spread over the case's range by ratio."""
    n, lo, hi = case["scenes"], case["min_width"], case["max_width"]
    widths = [int(lo * (hi / lo) ** (k / max(1, n - 1))) for k in range(n)]
    return [(w, w * 9 // 16) for w in widths]


class State:
    """What one program holds; closing order matters (an animation before its context)."""

    def __init__(self, case: dict, seed: int):
        self.case, self.animation, self.renderers = case, None, []
        self.frame_index = seed % 1000

    def renderer(self) -> GpuRenderer:
        self.renderers.append(GpuRenderer(0))
        return self.renderers[-1]

    def __del__(self):
        if self.animation is not None:
            self.animation.close()
        for r in self.renderers:
            r.close()


def prepare(case: dict, seed: int) -> State:
    st = State(case, seed)
    kind = case["kind"]
    if kind == "train":
        r = st.renderer()
        st.samples = _training_samples(case["samples"], seed)
        r.guide_set_params(guiding_eval.initial_params(seed), ROOM_BOUNDS)
    elif kind == "batch":
        scenes = configs.uneven_batch(seed % 100003, count=case["scenes"], samples=case["spp"],
                                      max_bounces=case["bounces"], environment=_sky(), min_width=case["min_width"],
                                      max_width=case["max_width"])
        for s, (w, h) in zip(scenes, _batch_sizes(case)):
            s.width, s.height = w, h
            st.renderer().upload(scene_to_gpu(s))
        st.out = [_pinned(s.height, s.width, 4) for s in scenes]
    elif kind == "animation":
        world = configs.BallisticAnimation(seed, case["width"], case["height"], case["spp"], case["bounces"],
                                           frames=48, environment=_sky())
        r = st.renderer()
        first = scene_to_gpu(world.scene(0))
        r.upload(first)
        st.animation = Animation(r, first, update_lights=True, rebuild=case["rebuild"])
        st.frame = scene_to_gpu(world.scene(1 + seed % 47))
        st.out = _pinned(case["height"], case["width"], 4, dtype=torch.uint8)
    else:
        r = st.renderer()
        scene = _scene(case, seed)
        st.data = scene_to_gpu(scene)
        if case.get("watertight"):
            r.set_triangle_test("watertight")
        r.upload(st.data)
        if kind == "hits":
            st.rays = configs.parity_rays(scene, case["rays"], seed)
            if not case["host"]:
                st.rays = torch.from_numpy(st.rays).cuda()
                st.prim = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
                st.t = torch.empty(case["rays"], dtype=torch.float32, device="cuda")
                torch.cuda.synchronize()
        elif kind == "guided":
            r.guide_set_params(guiding_eval.initial_params(seed), configs.scene_bounds(scene))
        if kind == "edit":
            st.out = _pinned(scene.height, scene.width, 4, dtype=torch.uint8)
        elif "width" in case:
            st.out = _pinned(scene.height, scene.width, 4)
    return st


def run(st: State):
    case, r = st.case, st.renderers[0]
    kind = case["kind"]
    if kind == "hits":
        if case["host"]:
            return r.trace_closest(st.rays)
        r.trace_closest_device(st.rays.data_ptr(), case["rays"], st.prim.data_ptr(), st.t.data_ptr())
        return st.prim, st.t
    if kind == "frame":
        r.render(frame_index=st.frame_index, keep_moments=case["moments"])
        return r.readback_sums(moments=True) if case["moments"] else r.readback(st.out)
    if kind == "progressive":
        for k in range(case["batches"]):
            r.render(samples=case["spp"], frame_index=st.frame_index + k, accumulate=k > 0)
        return r.readback_sums()[0]
    if kind == "guided":
        r.render(frame_index=st.frame_index, guiding=True, guide_record=int(case["record"]))
        return r.readback(st.out)
    if kind == "edit":
        r.upload(st.data)
        r.render(frame_index=st.frame_index)
        return r.readback_rgba8(out=st.out)
    if kind == "batch":
        render_batch(st.renderers, frame_index=st.frame_index)
        return [x.readback(o) for x, o in zip(st.renderers, st.out)]
    if kind == "animation":
        return st.animation.frame(st.frame, st.frame_index, st.out)
    grad, loss = r.guide_loss_grad(st.samples)
    return grad, loss


# ------------------------------------------------------------------------------------ work
# Rays per path (extension and shadow rays) of each scene at 8 bounces; fewer bounces take fewer.
RAYS_PER_PATH = {"small": 3.9, "mixed": 2.7, "room": 10.9, "mesh": 3.7}


def _trace_flops(rays: float, prims: int) -> float:
    """One descent per ray of a binary hierarchy with leaves of about two primitives: two box tests of
    18 operations per level, then two primitive tests of 50."""
    return rays * (max(1.0, math.log2(max(prims, 4) / 2)) * 36 + 100)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        # Forward, activation gradients and weight gradients of an 80-64-64-64-32 network.
        return {"bytes": 40 * case["samples"] + 2 * 4 * 15584, "flops": 3 * 30080 * case["samples"]}
    if kind == "hits":
        return {"bytes": 32 * case["rays"] + min(80 * case["prims"], 80 * case["rays"]),
                "flops": _trace_flops(case["rays"], case["prims"])}
    if kind == "batch":
        pixels = sum(w * h for w, h in _batch_sizes(case))
        return {"bytes": 16 * pixels + case["scenes"] * (80 * 6000 + 16 * 1024 * 512),
                "flops": _trace_flops(pixels * case["spp"] * 3.0, 6000)}
    pixels = case["width"] * case["height"]
    paths = pixels * case["spp"] * case.get("batches", 1)
    prims = case.get("prims", 834)
    rays = RAYS_PER_PATH[case.get("scene", "mixed")] * min(1.0, case["bounces"] / 8 + 0.3)
    out = {"edit": 4, "animation": 4, "progressive": 24}.get(kind, 48 if case.get("moments") else 16)
    return {"bytes": out * pixels + 80 * prims + 16 * 1024 * 512, "flops": _trace_flops(paths * rays, prims)}


# ------------------------------------------------------------------------------------ 64-bit values
def exact(case: dict, seed: int):
    if case["kind"] == "hits" and case["rays"] * case["prims"] <= 3e9:
        return None, _closest_64(_scene(case, seed), configs.parity_rays(_scene(case, seed), case["rays"], seed))
    if case["kind"] == "train":
        return _gradient_64(_training_samples(case["samples"], seed), guiding_eval.initial_params(seed))
    return None


def _closest_64(scene, rays: np.ndarray, tmin: float = 0.001) -> torch.Tensor:
    """Distance of the closest hit of every ray by testing every primitive (inf for a miss)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tmin = float(np.float32(tmin))
    d64 = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(dev)  # noqa: E731
    tri = d64(scene.triangles)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    inf = torch.tensor(math.inf, dtype=torch.float64, device=dev)
    best = []
    step = max(1, int(4e6 / max(1, len(v0))))
    for k in range(0, len(rays), step):
        o, d = d64(rays[k:k + step, :3])[:, None], d64(rays[k:k + step, 3:])[:, None]
        p = torch.linalg.cross(d.expand(-1, len(v0), -1), e2[None].expand(len(d), -1, -1))
        det = (e1[None] * p).sum(-1)
        s = o - v0[None]
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(len(d), -1, -1))
        v = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin)
        near = torch.where(ok, t, inf).amin(dim=1)
        if scene.sphere_count:
            oc = o - d64(scene.sphere_centers)[None]
            a, hb = (d * d).sum(-1), (oc * d).sum(-1)
            c = (oc * oc).sum(-1) - d64(scene.sphere_radii)[None] ** 2
            disc = hb * hb - a * c
            root = disc.clamp_min(0).sqrt()
            for t in ((-hb + root) / a, (-hb - root) / a):
                near = torch.minimum(near, torch.where((disc >= 0) & (t >= tmin), t, inf).amin(dim=1))
        best.append(near)
    return torch.cat(best)


def _gradient_64(samples: np.ndarray, flat: np.ndarray):
    """Gradient and value of the mean weighted negative log-likelihood of the 8-lobe mixture."""
    w = torch.from_numpy(flat.astype(np.float64)).requires_grad_()
    s = torch.from_numpy(samples.astype(np.float64))
    q = (s[:, :3] - torch.tensor(ROOM_BOUNDS[:3], dtype=torch.float64)) * ROOM_BOUNDS[3]
    ang = math.pi * q[:, :, None] * 2.0 ** (torch.arange(12, dtype=torch.float64) / 2)
    enc = torch.stack([ang.sin(), ang.cos()], dim=-1).reshape(len(s), 72)
    x = torch.cat([enc, s[:, 3:6], torch.zeros(len(s), 5, dtype=torch.float64)], dim=1)
    at = 0
    for k, (o, i) in enumerate([(64, 80), (64, 64), (64, 64), (32, 64)]):
        weight, bias = w[at:at + o * i].reshape(o, i), w[at + o * i:at + o * i + o]
        x = x @ weight.T + bias
        x = x.relu() if k < 3 else x
        at += o * i + o
    a, b, c, d = x.reshape(-1, 8, 4).unbind(-1)
    kappa, ct, phi = b.clamp(-2, 7).exp(), c.tanh(), math.pi * d.tanh()
    sine = (1 - ct * ct).clamp_min(0).sqrt()
    mu = torch.stack([sine * phi.cos(), sine * phi.sin(), ct], dim=-1)
    cos = (mu * s[:, None, 6:9]).sum(-1)
    lobe = kappa.log() - math.log(2 * math.pi) - torch.log1p(-(-2 * kappa).exp()) + kappa * (cos - 1)
    loss = -(s[:, 9] * torch.logsumexp(a.log_softmax(-1) + lobe, dim=-1)).mean()
    loss.backward()
    return w.grad, float(loss.detach())
