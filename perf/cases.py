"""Workloads the renderer is measured on: what a program that uses the package calls, from the smallest preview
to a full-HD ReSTIR sequence, over scenes of 36 to 8.4 million triangles.

Sizes follow the package's own configurations (the closed-box room at 256x256 with 16 samples, the instanced
scene at 1920x1080 with 4 samples and 8 bounces, the terrain at 1280x720 with 8 samples and 6 bounces, the
batched and served request mixes) and step away from them to odd and ragged ones.  Every case goes through the
public entry points of ``CudaWavefrontRenderer``.

Renders are Monte Carlo estimates whose random numbers are keyed by (pixel, sample, bounce, frame): the same case
and seed give the same paths, so two correct builds differ only by how rounding moves single decisions (a lobe, a
reservoir, an edge hit).
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import ordinarylight_b200 as ol
from ordinarylight_b200 import CudaWavefrontRenderer, scenes, workloads
from ordinarylight_b200.packing import pack_scene
from ordinarylight_b200.renderers.cuda import RenderRequest

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # The smallest call: an editor's thumbnail of a tiny scene, one sample, an odd width.
        dict(name="room_preview", kind="room", mode="production", width=161, height=90, spp=1, bounces=4),
        # The closed-box room at its configured size: reference-compatible transport, 16 samples.
        dict(name="room_reference", kind="room", mode="reference_compatible", width=256, height=256, spp=16, bounces=4),
        # The headline workload: a frame sequence of the instanced scene (1,049,602 triangles) with ReSTIR and its
        # temporal reuse, left on the device for a denoiser or an encoder.
        dict(name="spheres_restir_1080p", kind="spheres", instances=64, width=1920, height=1080, spp=4, bounces=8,
             restir=True),
        # An ordinary viewport of ragged size with plain next-event estimation, one sample a frame.
        dict(name="spheres_nee_ragged", kind="spheres", instances=23, width=1003, height=601, spp=1, bounces=6,
             restir=False),
        # The terrain with its delta-tracked medium, sky and sun: the largest geometry, 8,380,418 triangles.
        dict(name="terrain_volume_720p", kind="terrain", grid=2048, width=1280, height=720, spp=8, bounces=6,
             volume=True),
        # An asset viewer: textured, normal-mapped and glass objects under panels and a point light, with ReSTIR.
        dict(name="textured_restir_540p", kind="textured", width=960, height=540, spp=2, bounces=5, restir=True),
        # Scientific volumes beside surfaces: the reference's emission-absorption ray march, two media.
        dict(name="march_volumes", kind="march", width=320, height=180, spp=2, bounces=3),
        # A render farm's batch: jobs of uneven size and sample count over several resident scenes, images on the host.
        dict(name="batch_mixed", kind="batch", jobs=16, scale=1.0),
        # A serving loop's burst: small requests queued together and collected as they finish.
        dict(name="serve_burst", kind="serve", jobs=24, scale=0.5),
        # Ray queries of a program of its own (picking, occlusion baking): closest hits, then visibility.
        dict(name="query_rays", kind="query", instances=64, segments=128, rays=600_001),
        # A streamed level: a new mesh of 2.1 million triangles is made resident and its first rays are traced.
        dict(name="load_terrain", kind="load", grid=1025, rays=20_000),
        # An animation: an object deforms and others move each frame, the scene is updated in place and rendered.
        dict(name="animate_spheres", kind="animate", instances=48, segments=96, width=640, height=360, spp=1,
             bounces=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, pixels):
    """A width and a height of at most `pixels` pixels, odd ones among them."""
    w = _log_int(rng, lo, hi)
    return w, max(16, min(int(w * rng.uniform(0.5, 1.0)), pixels // w))


def draw(rng):
    kind = rng.choice(("room", "room", "spheres", "spheres", "terrain", "textured", "march", "batch", "serve",
                       "query", "load", "animate"))
    if kind == "room":
        w, h = _size(rng, 96, 1024, 1 << 19)
        return dict(kind=kind, mode=rng.choice(("production", "reference_compatible")), width=w, height=h,
                    spp=rng.choice((1, 2, 4, 16)), bounces=rng.randint(2, 8))
    if kind == "spheres":
        w, h = _size(rng, 160, 1920, 1920 * 1080)
        return dict(kind=kind, instances=_log_int(rng, 4, 128), width=w, height=h, spp=rng.choice((1, 2, 4)),
                    bounces=rng.randint(3, 8), restir=rng.random() < 0.5)
    if kind == "terrain":
        w, h = _size(rng, 160, 1280, 1280 * 720)
        return dict(kind=kind, grid=rng.choice((300, 777, 1201)), width=w, height=h, spp=rng.choice((1, 2, 4, 8)),
                    bounces=rng.randint(2, 6), volume=rng.random() < 0.6)
    if kind == "textured":
        w, h = _size(rng, 160, 1280, 1280 * 720)
        return dict(kind=kind, width=w, height=h, spp=rng.choice((1, 2, 4)), bounces=rng.randint(2, 6),
                    restir=rng.random() < 0.5)
    if kind == "march":
        w, h = _size(rng, 64, 480, 480 * 270)
        return dict(kind=kind, width=w, height=h, spp=rng.choice((1, 2)), bounces=rng.randint(1, 4))
    if kind in ("batch", "serve"):
        return dict(kind=kind, jobs=rng.randint(4, 24), scale=round(rng.uniform(0.25, 1.0), 3))
    if kind == "query":
        return dict(kind=kind, instances=_log_int(rng, 2, 64), segments=rng.choice((16, 32, 64, 128)),
                    rays=_log_int(rng, 1_000, 1_000_000))
    if kind == "load":
        return dict(kind=kind, grid=_log_int(rng, 100, 1025), rays=_log_int(rng, 500, 20_000))
    w, h = _size(rng, 160, 960, 960 * 540)
    return dict(kind=kind, instances=_log_int(rng, 4, 64), segments=rng.choice((32, 64, 96)), width=w, height=h,
                spp=1, bounces=rng.randint(2, 6))


# ---------------------------------------------------------------------------
# scenes (geometry that a program has in hand; what is costly to make and the same for every seed is kept)
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=8)
def _heights(grid):
    return scenes.fbm_heightfield(grid, seed=3)


def _grid_normals(heights, spacing):
    gz, gx = np.gradient(heights.astype(np.float32), spacing)
    n = np.stack([-gx, np.ones_like(gx), -gz], -1).reshape(-1, 3)
    return n / np.linalg.norm(n, axis=1, keepdims=True)


def _terrain_scene(heights, volume_size=0):
    scene = ol.Scene()
    spacing = 512.0 / heights.shape[0]
    v, i = scenes.grid_mesh(heights, spacing)
    n = _grid_normals(heights, spacing)
    tangents = np.zeros((len(v), 4), np.float32)
    tangents[:, 0] = n[:, 1]
    tangents[:, 1] = -n[:, 0]
    tangents[:, 3] = 1.0
    ground = scene.create_mesh(v, i, ol.Material(base_color=(0.4, 0.4, 0.4)), normals=n, tangents=tangents,
                               name="terrain")
    scene.add_instance(ground)
    scene.set_environment(ol.EnvironmentLight(color=(1.0, 1.0, 1.0), intensity=1.0))
    scene.add_light(ol.DirectionalLight(direction=(-0.4, -1.0, 0.3), color=(1.0, 0.95, 0.85), intensity=3.0))
    if volume_size:
        xf = ol.Transform.translation((-60.0, 20.0, -60.0)) @ ol.Transform.scale(120.0)
        scene.add_volume(scenes.fbm_volume(volume_size, seed=4), ol.VolumeMaterial(sigma_t_scale=0.5, albedo=0.9),
                         transform=xf, name="cloud")
    camera = ol.PerspectiveCamera(position=(0.0, 120.0, -300.0), target=(0.0, 0.0, 0.0), vertical_fov_degrees=50.0)
    return scene, camera


@functools.lru_cache(maxsize=4)
def _terrain(grid, volume):
    scene, camera = _terrain_scene(_heights(grid), 128 if volume else 0)
    return pack_scene(scene), camera


def _noise_texture(rng, size, low, high):
    """A smooth RGBA8 texture of two octaves of value noise."""
    coarse = rng.uniform(low, high, (size // 16, size // 16, 3))
    fine = rng.uniform(low, high, (size, size, 3))
    px = 0.7 * np.kron(coarse, np.ones((16, 16, 1))) + 0.3 * fine
    return np.concatenate([px, np.full((size, size, 1), 255.0)], -1).astype(np.uint8)


def _textured_scene(seed):
    rng = np.random.default_rng(seed)
    scene = ol.Scene()
    albedo = ol.Texture(_noise_texture(rng, 512, 40, 230))
    rough = ol.Texture(_noise_texture(rng, 256, 30, 255))
    normal = _noise_texture(rng, 256, 108, 148)
    normal[..., 2] = 240
    normal = ol.Texture(normal, wrap_s="mirror", wrap_t="mirror")
    quad = np.array([[-8, 0, -8], [-8, 0, 8], [8, 0, 8], [8, 0, -8]], np.float32)
    floor = scene.create_mesh(quad, np.array([[0, 1, 2], [0, 2, 3]], np.uint32),
                              ol.Material(base_color=(0.9, 0.9, 0.9), roughness=0.9, base_color_texture=albedo,
                                          metallic_roughness_texture=rough, normal_texture=normal),
                              normals=np.tile([0.0, 1.0, 0.0], (4, 1)).astype(np.float32), texcoords=quad[:, [0, 2]] * 0.2)
    scene.add_instance(floor)
    v, i, n = scenes.uv_sphere(96, 49)
    uv = np.stack([np.arctan2(v[:, 2], v[:, 0]) / (2 * math.pi) + 0.5, np.arccos(np.clip(v[:, 1], -1, 1)) / math.pi], -1)
    ball = scene.create_mesh(v, i, ol.Material(), normals=n, texcoords=(uv * 3.0).astype(np.float32))
    placed, materials = [], []
    for k in range(24):
        x, z = (k % 6) * 2.2 - 5.5, (k // 6) * 2.2 - 3.3
        placed.append(ol.Transform.translation((x + rng.uniform(-0.3, 0.3), 0.8, z)) @ ol.Transform.scale(0.8))
        if k % 6 == 5:
            materials.append(ol.Material(base_color=(0.95, 0.97, 1.0), roughness=0.05, transmission=1.0, ior=1.5))
        else:
            materials.append(ol.Material(base_color=tuple(float(c) for c in rng.uniform(0.4, 1.0, 3)), roughness=0.7,
                                         metallic=float(k % 3 == 0), base_color_texture=albedo if k % 2 else None,
                                         metallic_roughness_texture=rough, normal_texture=normal if k % 4 else None))
    scene.add_instances(ball, placed, materials=materials)
    for x in (-4.0, 0.0, 4.0):
        panel = np.array([[x - 1, 6, -1], [x + 1, 6, -1], [x + 1, 6, 1], [x - 1, 6, 1]], np.float32)
        scene.add_mesh(panel, np.array([[0, 1, 2], [0, 2, 3]], np.uint32),
                       ol.Material(base_color=(0.0, 0.0, 0.0), emission=(9.0, 8.0, 7.0)))
    scene.add_light(ol.PointLight(position=(-3.0, 4.0, -6.0), color=(1.0, 0.9, 0.8), intensity=20.0))
    camera = ol.PerspectiveCamera(position=(0.0, 4.5, -10.0), target=(0.0, 0.5, 0.0), vertical_fov_degrees=45.0)
    return scene, camera


def _march_scene(seed):
    scene, camera = scenes.box_room()
    glow = ol.Texture1D(np.array([[0.0, 0.0, 0.0, 0.0], [1.0, 0.5, 0.2, 0.3], [0.4, 0.6, 1.0, 0.9]], np.float32))
    scene.add_volume(scenes.fbm_volume(64, seed=21 + seed % 1000, octaves=3),
                     ol.VolumeMaterial(transfer_function=glow, density_scale=0.8, emission_scale=0.5, step_size=0.02,
                                       scattering_scale=1.0, phase_function="henyey_greenstein", anisotropy=0.3,
                                       scattering_orders=2),
                     transform=ol.Transform.translation((-0.7, 0.2, -0.6)))
    mist = ol.Texture1D(np.array([[0.0, 0.0, 0.0, 0.0], [0.2, 0.9, 0.3, 0.6], [0.9, 0.9, 0.9, 0.2]], np.float32))
    scene.add_volume(scenes.fbm_volume(48, seed=22 + seed % 1000, octaves=3),
                     ol.VolumeMaterial(transfer_function=mist, density_scale=0.6, emission_scale=0.8, step_size=0.015),
                     transform=ol.Transform.translation((-0.25, 0.45, -0.35)) @ ol.Transform.scale(0.8))
    scene.add_light(ol.PointLight(position=(0.0, 1.7, -0.4), color=(1.0, 0.9, 0.7), intensity=2.0))
    return scene, camera


@functools.lru_cache(maxsize=1)
def _mixed_scenes():
    room = scenes.box_room(tessellation=40)
    spheres = scenes.instanced_spheres(seed=9, instances=16, emitters=256)
    packed, camera = _terrain(300, True)
    return [("room", *room), ("spheres", *spheres), ("terrain", packed, camera)]


def _requests(case, rng):
    """Requests over the three kinds of scene, sizes and samples as the served and batched mixes draw them."""
    out = []
    shapes = ((128, 128), (256, 256), (512, 512), (640, 360), (1280, 720))
    for k in range(case["jobs"]):
        kind, scene, camera = _mixed_scenes()[k % 3]
        w, h = shapes[(k * 7 + 2) % 5]
        spp = (1, 4, 16)[(k // 2) % 3] if w * h <= 512 * 512 else 1
        out.append(RenderRequest(scene, workloads.seeded_camera(camera, rng), max(16, int(w * case["scale"])),
                                 max(16, int(h * case["scale"])), samples=spp, frame_index=int(rng.integers(1 << 16)),
                                 max_bounces=workloads.CONFIG_BOUNCES[kind]))
    return out


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    frame = int(rng.integers(1 << 20))
    if kind in ("batch", "serve"):
        renderer = CudaWavefrontRenderer()
        requests = _requests(case, rng)
        for request in requests:
            renderer.resident_scene(request.scene)
        return dict(case=case, renderer=renderer, requests=requests)
    if kind == "query":
        scene, _ = scenes.instanced_spheres(seed=int(rng.integers(1 << 20)), instances=case["instances"],
                                            segments=case["segments"], bands=case["segments"] // 2 + 1, emitters=64)
        n = case["rays"]

        def rays():
            d = rng.standard_normal((n, 3))
            return (rng.uniform(-22.0, 22.0, (n, 3)).astype(np.float32),
                    (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))

        o, d = rays()
        so, sd = rays()
        renderer = CudaWavefrontRenderer()
        renderer.trace_closest(scene, o[:1], d[:1])   # the scene is resident
        return dict(case=case, renderer=renderer, scene=scene, o=o, d=d, so=so, sd=sd,
                    far=rng.uniform(1.0, 40.0, n).astype(np.float32))
    if kind == "load":
        shift = rng.integers(0, case["grid"], 2)
        heights = np.ascontiguousarray(np.roll(_heights(case["grid"]), tuple(int(k) for k in shift), (0, 1)))
        n = case["rays"]
        o = np.stack([rng.uniform(-250, 250, n), np.full(n, 200.0), rng.uniform(-250, 250, n)], -1).astype(np.float32)
        d = np.stack([rng.uniform(-0.5, 0.5, n), np.full(n, -1.0), rng.uniform(-0.5, 0.5, n)], -1)
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        renderer = CudaWavefrontRenderer()
        renderer.replace_scene(_terrain(300, False)[0])   # the level that the new one replaces
        return dict(case=case, renderer=renderer, scene=pack_scene(_terrain_scene(heights)[0]), o=o, d=d)

    options = dict(samples_per_pixel=case["spp"], max_bounces=case["bounces"], mode=case.get("mode", "production"),
                   restir=case.get("restir", False))
    state = dict(case=case, frame=frame)
    if kind == "room":
        scene, camera = scenes.box_room()
    elif kind == "spheres":
        scene, camera = scenes.instanced_spheres(seed=int(rng.integers(1 << 20)), instances=case["instances"])
    elif kind == "terrain":
        scene, camera = _terrain(case["grid"], case["volume"])
    elif kind == "textured":
        scene, camera = _textured_scene(int(rng.integers(1 << 20)))
    elif kind == "march":
        scene, camera = _march_scene(int(rng.integers(1 << 20)))
        options["mode"] = "reference_compatible"
    else:
        scene, camera = scenes.instanced_spheres(seed=int(rng.integers(1 << 20)), instances=case["instances"],
                                                 segments=case["segments"], bands=case["segments"] // 2 + 1,
                                                 emitters=128)
        v, i, n = scenes.uv_sphere(case["segments"], case["segments"] // 2 + 1, radius=4.0)
        flag = scene.create_mesh(v, i, ol.Material(base_color=(0.7, 0.3, 0.2), roughness=0.4), normals=n,
                                 deformable=True)
        scene.add_instance(flag)
        state["flag"] = flag
        state["shapes"] = [(v * (1.0 + 0.2 * np.sin(3.0 * v[:, 1:2] + k))).astype(np.float32) for k in range(4)]
        state["normals"] = n
        movers = [m for m in scene.visible_meshes if len(m.indices) > 64][:8]
        state["movers"] = movers
        poses = []
        for k in range(4):
            row = []
            for m in movers:
                xf = np.array(m.transform.matrix, copy=True)
                xf[:3, 3] += (0.3 * math.sin(k), 0.2 * k, 0.3 * math.cos(k))
                row.append(ol.Transform(xf))
            poses.append(row)
        state["poses"] = poses
    renderer = CudaWavefrontRenderer(**options)
    camera = workloads.seeded_camera(camera, rng)
    state.update(renderer=renderer, scene=scene, camera=camera)
    if kind in ("spheres", "terrain", "animate"):
        state["out"] = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
    renderer.render_frame(scene, camera, 16, 16, samples=1)   # the scene is resident
    return state


def run(state):
    case, r = state["case"], state["renderer"]
    kind = case["kind"]
    if kind == "batch":
        return r.render_batch(state["requests"])
    if kind == "serve":
        for request in state["requests"]:
            r.submit(request)
        images = {}
        while r.queued_tickets():
            for ticket, image in r.serve_step():
                images[ticket] = image
        return [images[ticket] for ticket in sorted(images)]
    if kind == "query":
        inst, prim, t, bary = r.trace_closest(state["scene"], state["o"], state["d"])
        seen = r.trace_occluded(state["scene"], state["so"], state["sd"], state["far"])
        return dict(instance=inst.view(np.int32), primitive=prim, t=t, bary=bary, occluded=seen)
    if kind == "load":
        r.replace_scene(state["scene"])
        inst, prim, t, bary = r.trace_closest(state["scene"], state["o"], state["d"])
        return dict(primitive=prim, t=t, bary=bary)
    w, h, scene, camera = case["width"], case["height"], state["scene"], state["camera"]
    frame = state["frame"]
    state["frame"] = frame + 1
    if kind == "animate":
        pose = frame % 4
        scene.update_instance_transforms(state["movers"], state["poses"][pose])
        scene.update_mesh_resource(state["flag"], vertices=state["shapes"][pose], normals=state["normals"])
    if "out" in state:
        return r.render_frame_into(scene, camera, w, h, state["out"], frame_index=frame)
    return r.render_frame(scene, camera, w, h, frame_index=frame)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

# Geometry as it is given: three indices and half a vertex (position, normal) a triangle.
_TRIANGLE_BYTES = 24.0
# Operations of one ray through a hierarchy of n triangles: about log2(n) box pairs and two triangle tests, and of one
# vertex: the BSDF, a light and a sampled direction.
_VERTEX_FLOPS = 300.0


def _ray_flops(triangles):
    return 30.0 * math.log2(max(triangles, 2)) + 100.0


def _triangles(case):
    kind = case["kind"]
    if kind == "room" or kind == "march":
        return 36
    if kind == "spheres":
        return case["instances"] * 16384 + 1026
    if kind in ("terrain", "load"):
        return 2 * (case["grid"] - 1) ** 2
    if kind == "textured":
        return 24 * 9216 + 8
    if kind in ("batch", "serve"):
        return 100_000
    return case["instances"] * case["segments"] ** 2


def work(case):
    kind, n = case["kind"], _triangles(case)
    if kind == "query":
        return {"bytes": case["rays"] * (24.0 + 20.0 + 28.0 + 1.0), "flops": 2.0 * case["rays"] * _ray_flops(n)}
    if kind == "load":
        return {"bytes": n * (_TRIANGLE_BYTES + 108.0 + 64.0), "flops": n * math.log2(n) * 20.0}
    if kind in ("batch", "serve"):
        paths = image = 0.0
        for k in range(case["jobs"]):
            w, h = ((128, 128), (256, 256), (512, 512), (640, 360), (1280, 720))[(k * 7 + 2) % 5]
            spp = (1, 4, 16)[(k // 2) % 3] if w * h <= 512 * 512 else 1
            pixels = w * h * case["scale"] ** 2
            image += pixels
            paths += pixels * spp
        return {"bytes": 16.0 * image + n * _TRIANGLE_BYTES, "flops": paths * 3.0 * (2.0 * _ray_flops(n) + _VERTEX_FLOPS)}
    pixels = case["width"] * case["height"]
    depth = min(case["bounces"], 3.0)   # paths leave the scene or end after a few vertices
    flops = pixels * case["spp"] * depth * (2.0 * _ray_flops(n) + _VERTEX_FLOPS)
    if kind == "march":
        flops += pixels * case["spp"] * depth * 100.0 * 80.0   # about a hundred steps a segment
    return {"bytes": 16.0 * pixels + n * _TRIANGLE_BYTES, "flops": flops}


def tolerance(case):
    """About four times what the same sources give with every multiply-add rounded twice instead of once.  A render
    differs where that turns a lobe, a reservoir or a survival the other way; the room's reference-compatible
    transport makes no such choice but its hits."""
    kind = case["kind"]
    if kind == "query":
        # float32 distances and barycentrics; a ray that meets an edge or a tie may report the neighbour
        return {"rel": 0.025, "max": 0.99, "differ": 1e-4}
    if kind == "load":
        return {"rel": 1e-4, "max": 0.5, "differ": 1e-4}
    if case.get("mode") == "reference_compatible":
        return {"rel": 2.5e-4, "max": 0.06}
    if kind == "march":
        return {"rel": 2e-3, "max": 0.8}
    return {"rel": 0.015, "max": 0.99}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _world_triangles(scene, device):
    """(n, 3, 3) vertices, (n, 3) base colours and emissions of the visible meshes, in order."""
    tris, base, emission = [], [], []
    for m in scene.visible_meshes:
        x = np.asarray(m.transform.matrix, np.float64)
        v = np.asarray(m.vertices, np.float64) @ x[:3, :3].T + x[:3, 3]
        tris.append(v[np.asarray(m.indices)])
        base.append(np.tile(m.material.base_color, (len(m.indices), 1)))
        emission.append(np.tile(m.material.emission, (len(m.indices), 1)))
    return [torch.as_tensor(np.concatenate(a), dtype=torch.float64, device=device) for a in (tris, base, emission)]


def _nearest(o, d, tris, t_min, t_max=None):
    """Nearest hit of every ray (Moeller and Trumbore 1997) among all triangles: t (inf: none), index, b1, b2."""
    n = len(o)
    best = torch.full((n,), math.inf, dtype=torch.float64, device=o.device)
    which = torch.full((n,), -1, dtype=torch.int64, device=o.device)
    b1, b2 = torch.zeros_like(best), torch.zeros_like(best)
    chunk = max(1, (1 << 25) // max(n, 1))
    for first in range(0, len(tris), chunk):
        v0 = tris[first:first + chunk, 0][None]
        e1 = tris[first:first + chunk, 1][None] - v0
        e2 = tris[first:first + chunk, 2][None] - v0
        dd = d[:, None, :]
        p = torch.linalg.cross(dd.expand(-1, e2.shape[1], -1), e2.expand(n, -1, -1))
        det = (e1 * p).sum(-1)
        inv = 1.0 / det
        s = o[:, None, :] - v0
        u = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1.expand(n, -1, -1))
        v = (dd * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > t_min)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        tc, k = t.min(1)
        nearer = tc < best
        best = torch.where(nearer, tc, best)
        which = torch.where(nearer, k + first, which)
        b1 = torch.where(nearer, u.gather(1, k[:, None])[:, 0], b1)
        b2 = torch.where(nearer, v.gather(1, k[:, None])[:, 0], b2)
    return best, which, b1, b2


_M32 = 0xFFFFFFFF


def _hash(v):
    v = v & _M32
    v = v ^ (v >> 16)
    v = (v * 0x7FEB352D) & _M32
    v = v ^ (v >> 15)
    v = (v * 0x846CA68B) & _M32
    return v ^ (v >> 16)


def _draw_uniform(state):
    state = (state * 747796405 + 2891336453) & _M32
    word = (((state >> ((state >> 28) + 4)) ^ state) * 277803737) & _M32
    return ((word >> 22) ^ word).double() / 4294967296.0, state


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _exact_room(case, state):
    """The reference-compatible transport of the closed-box room, path by path with the same random numbers."""
    dev = _device()
    tris, base, emission = _world_triangles(state["scene"], dev)
    normals = _unit(torch.linalg.cross(tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]))
    w, h, cam = case["width"], case["height"], state["camera"]
    pos = torch.tensor(cam.position, dtype=torch.float64, device=dev)
    forward = _unit(torch.tensor(cam.target, dtype=torch.float64, device=dev) - pos)
    right = _unit(torch.linalg.cross(forward, torch.tensor(cam.up, dtype=torch.float64, device=dev)))
    up = torch.linalg.cross(right, forward)
    half = math.tan(math.radians(cam.vertical_fov_degrees) / 2.0)
    pixel = torch.arange(w * h, device=dev)
    key = 1 + state["frame"]   # the renderer's seed and the frame
    frame = _hash(torch.tensor(key, device=dev))
    image = torch.zeros((w * h, 3), dtype=torch.float64, device=dev)
    for sample in range(case["spp"]):
        seed = _hash(_hash(pixel ^ frame) ^ _hash(torch.tensor(sample + 1, device=dev)))
        j1 = _hash(seed)
        jx, jy = j1.double() / 4294967296.0, _hash(j1).double() / 4294967296.0
        nx = ((pixel % w).double() + jx) / w * 2.0 - 1.0
        ny = 1.0 - (torch.div(pixel, w, rounding_mode="floor").double() + jy) / h * 2.0
        d = _unit(forward + nx[:, None] * (half * w / h) * right + ny[:, None] * half * up)
        o = pos.expand_as(d)
        weight = torch.ones_like(d)
        alive = torch.ones(w * h, dtype=torch.bool, device=dev)
        for bounce in range(case["bounces"]):
            t, k, _, _ = _nearest(o, d, tris, 1e-4)
            hit = k >= 0
            blend = (0.5 * (d[:, 1:2] + 1.0)).clamp(0.0, 1.0)
            sky = (torch.tensor([0.8, 0.8, 0.8], dtype=torch.float64, device=dev) * (1.0 - blend)
                   + torch.tensor([0.2, 0.4, 0.9], dtype=torch.float64, device=dev) * blend)
            kk = k.clamp(min=0)
            light = torch.where(hit[:, None], emission[kk], sky)
            image += torch.where(alive[:, None], weight * light, torch.zeros_like(light))
            alive = alive & hit
            weight = weight * base[kk]
            n = normals[kk]
            n = torch.where((n * d).sum(-1, keepdim=True) > 0, -n, n)
            s = _hash(seed ^ _hash(torch.tensor((bounce * 0x9E3779B9 + 0x632BE5AB) & _M32, device=dev)))
            u1, s = _draw_uniform(s)
            u2, s = _draw_uniform(s)
            z = 1.0 - 2.0 * u1
            rad = (1.0 - z * z).clamp(min=0.0).sqrt()
            ball = torch.stack([rad * torch.cos(2 * math.pi * u2), rad * torch.sin(2 * math.pi * u2), z], -1)
            ball = torch.where((ball * n).sum(-1, keepdim=True) < 0, -ball, ball)
            o = o + d * torch.where(hit, t, torch.zeros_like(t))[:, None] + n * 1e-4
            d = _unit(n + ball)
    out = torch.zeros((h, w, 4), dtype=torch.float64, device=dev)
    out[..., :3] = (image / case["spp"]).reshape(h, w, 3)
    return out


def exact(case, seed):
    """Renders beyond the room's plain transport go through millions of triangles, lights and reservoirs: a 64-bit
    path by path computation of them takes far longer than 20 seconds."""
    if case["kind"] == "room" and case["mode"] == "reference_compatible":
        return _exact_room(case, prepare(case, seed))
    if case["kind"] in ("query", "load"):
        triangles = _triangles(case)
        if triangles * case["rays"] > 8e9:
            return None
        s = prepare(case, seed)
        dev = _device()
        if case["kind"] == "load":
            v = torch.as_tensor(s["scene"].vertices, dtype=torch.float64, device=dev).reshape(-1, 3)
            tris = v[torch.as_tensor(s["scene"].indices.astype(np.int64), device=dev).reshape(-1, 3)]
        else:
            tris = _world_triangles(s["scene"], dev)[0]
        o, d = (torch.as_tensor(s[k], dtype=torch.float64, device=dev) for k in ("o", "d"))
        t, k, b1, b2 = _nearest(o, d, tris, 1e-4)
        out = dict(primitive=None, t=t, bary=torch.stack([b1, b2], -1))
        return out if case["kind"] == "load" else dict(out, instance=None, occluded=None)
    return None
