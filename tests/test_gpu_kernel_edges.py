"""Kernel edges on the device: sizes and shapes where a kernel's split, its
shared stack or a dispatch rule can go wrong, against brute force, a library
sort or the oracle."""

from __future__ import annotations

import numpy as np
import pytest

import ordinarylight_b200 as ol
from ordinarylight_b200 import CudaWavefrontRenderer, _native

pytestmark = pytest.mark.gpu


def _mesh_scene(vertices, indices, normal=(0.0, 0.0, 1.0)):
    """A scene of one mesh (its own normals and tangents, so making it is quick)."""
    scene = ol.Scene()
    n = np.tile(np.asarray(normal, np.float32), (len(vertices), 1))
    tangents = np.tile(np.float32([1.0, 0.0, 0.0, 1.0]), (len(vertices), 1))
    mesh = scene.create_mesh(np.asarray(vertices, np.float32), np.asarray(indices, np.uint32),
                             ol.Material(base_color=(0.5, 0.5, 0.5)), normals=n, tangents=tangents)
    scene.add_instance(mesh)
    return scene


@pytest.mark.parametrize("stack_depth", [16, 24, 32])
@pytest.mark.parametrize("rays", [1, 33, 5000, 40_000])
def test_deep_stacks_and_every_ray_count(native_library, cuda_device, stack_depth, rays):
    """20,000 parallel sheets: a ray through them meets all four boxes of every
    node, so its stack (three entries a level) runs past 16 shared entries into
    the overflow.  Half of the rays pass each sheet's box beside its triangle
    and visit the whole tree.  Ray counts below and above one ray per warp."""
    sheets = 20_000
    z = np.arange(sheets, dtype=np.float32)
    v = np.zeros((sheets, 3, 3), np.float32)
    v[:, 1, 0] = v[:, 2, 1] = 1.0
    v[:, :, 2] = z[:, None]
    scene = _mesh_scene(v.reshape(-1, 3), np.arange(3 * sheets).reshape(-1, 3))
    rng = np.random.default_rng(rays)
    xy = rng.uniform(0.05, 0.45, (rays, 2))
    outside = np.arange(rays) % 2 == 1
    xy[outside] += 0.5                        # x + y > 1: in the box, off the triangle
    start = rng.integers(-1, sheets - 1, rays) + 0.5
    o = np.column_stack([xy, start]).astype(np.float32)
    up = np.arange(rays) % 3 != 0
    d = np.zeros((rays, 3), np.float32)
    d[:, 2] = np.where(up, 1.0, -1.0)
    first = np.where(up, np.ceil(start), np.floor(start)).astype(np.int64)
    hit = ~outside & (first >= 0) & (first < sheets)
    with CudaWavefrontRenderer(stack_depth=stack_depth) as r:
        _inst, prim, t, _ = r.trace_closest(scene, o, d)
        np.testing.assert_array_equal(prim, np.where(hit, first, -1))
        np.testing.assert_array_equal(t, np.where(hit, 0.5, np.inf).astype(np.float32))
        far = np.full(rays, 1e9, np.float32)
        np.testing.assert_array_equal(r.trace_occluded(scene, o, d, far), hit)
        np.testing.assert_array_equal(r.trace_occluded(scene, o, d, np.full(rays, 0.25, np.float32)), np.zeros(rays, bool))


@pytest.mark.parametrize("instances,answered", [(100, True), (210, False)])
def test_rays_past_the_step_budget_are_errors_in_both_queries(native_library, cuda_device, instances, answered):
    """A ray beside the triangles of 20,000 sheets visits every node and leaf
    of the mesh, 20,000 to 26,700 steps, in each of its coincident instances: 100
    stay within the 4,194,304 steps a ray may take and 210 do not.  Neither
    query may answer for a ray that it did not finish."""
    sheets = 20_000
    v = np.zeros((sheets, 3, 3), np.float32)
    v[:, 1, 0] = v[:, 2, 1] = 1.0
    v[:, :, 2] = np.arange(sheets, dtype=np.float32)[:, None]
    scene = ol.Scene()
    vertices = v.reshape(-1, 3)
    mesh = scene.create_mesh(vertices, np.arange(3 * sheets).reshape(-1, 3), ol.Material(),
                             normals=np.tile(np.float32([0.0, 0.0, 1.0]), (len(vertices), 1)),
                             tangents=np.tile(np.float32([1.0, 0.0, 0.0, 1.0]), (len(vertices), 1)))
    scene.add_instances(mesh, [ol.Transform.translation((0.0, 0.0, 0.0))] * instances)
    o = np.float32([[0.75, 0.75, -1.0]])
    d = np.float32([[0.0, 0.0, 1.0]])
    far = np.full(1, 1e9, np.float32)
    with CudaWavefrontRenderer() as r:
        if answered:
            assert r.trace_closest(scene, o, d)[1][0] == -1
            assert not r.trace_occluded(scene, o, d, far)[0]
        else:
            with pytest.raises(RuntimeError, match="traversal"):
                r.trace_closest(scene, o, d)
            with pytest.raises(RuntimeError, match="traversal"):
                r.trace_occluded(scene, o, d, far)
            # the next query is answered
            assert r.trace_closest(scene, np.float32([[0.25, 0.25, -1.0]]), d)[2][0] == 1.0


def test_waiting_for_other_rays_spends_no_step_budget(native_library, cuda_device):
    """A ray through 160 coincident instances of 20,000 sheets takes about 3.5
    million of its 4,194,304 steps.  In one warp with four such rays, which set
    out elsewhere and meet their leaves at other steps, it is answered as it
    is alone.  The queue fills warps with 32 rays; the others miss the scene."""
    sheets, instances = 20_000, 160
    v = np.zeros((sheets, 3, 3), np.float32)
    v[:, 1, 0] = v[:, 2, 1] = 1.0
    v[:, :, 2] = np.arange(sheets, dtype=np.float32)[:, None]
    scene = ol.Scene()
    vertices = v.reshape(-1, 3)
    mesh = scene.create_mesh(vertices, np.arange(3 * sheets).reshape(-1, 3), ol.Material(),
                             normals=np.tile(np.float32([0.0, 0.0, 1.0]), (len(vertices), 1)),
                             tangents=np.tile(np.float32([1.0, 0.0, 0.0, 1.0]), (len(vertices), 1)))
    scene.add_instances(mesh, [ol.Transform.translation((0.0, 0.0, 0.0))] * instances)
    n = 2_000_000
    o = np.tile(np.float32([5.0, 5.0, -1.0]), (n, 1))
    d = np.tile(np.float32([0.0, 0.0, 1.0]), (n, 1))
    o[:5] = np.column_stack([np.full(5, 0.75), np.full(5, 0.75), np.arange(5) * 37.0 - 1.0])
    with CudaWavefrontRenderer() as r:
        assert np.all(r.trace_closest(scene, o, d)[1] == -1)
        assert not r.trace_occluded(scene, o, d, np.full(n, 1e9, np.float32)).any()


@pytest.mark.parametrize("extent", [(100.0, 1.0, 100.0), (0.0, 5.0, 1000.0), (1e-3, 1.0, 1e3), (0.0, 0.0, 0.0)])
def test_morton_cells_of_any_extent_build_a_valid_tree(native_library, cuda_device, extent):
    """Meshes above the host builder's limit whose extents differ by up to
    10^6, or vanish: the tree validates and rays that start beside their
    targets report the oracle's hits."""
    from oracle import production

    count = 140_000
    rng = np.random.default_rng(3)
    centre = rng.uniform(-0.5, 0.5, (count, 1, 3)) * np.asarray(extent)
    v = (centre + rng.uniform(-0.01, 0.01, (count, 3, 3))).astype(np.float32)
    scene = _mesh_scene(v.reshape(-1, 3), np.arange(3 * count).reshape(-1, 3))
    n = 4000
    aim = rng.integers(0, count, n)
    target = v[aim].astype(np.float64).mean(1)
    o = (target + 3.0 * rng.normal(size=(n, 3))).astype(np.float32)
    d = target - o
    dist = np.linalg.norm(d, axis=1)
    d = (d / dist[:, None]).astype(np.float32)
    with CudaWavefrontRenderer() as r:
        assert r.validate_bvh(scene) == 0
        _inst, prim, t, _ = r.trace_closest(scene, o, d)
    # a direction rounds by 1e-7 of the few units to a triangle 0.01 wide: all but slivers are hit, none is passed
    hit = prim >= 0
    assert hit.mean() > 0.99
    assert np.all(t[hit] <= dist[hit] * (1 + 1e-6) + 0.02)
    want, want_t = production.trace(scene, o, d)
    same = prim == want
    assert same.mean() > 0.995
    # another triangle only at the same distance, or where the ray passes an edge of the nearer of the two, each within
    # four roundings of the coordinates
    other = np.flatnonzero(~same)
    slack = 4 * np.spacing(np.abs(o[other]).max(1) + dist[other].astype(np.float32)).astype(np.float64)
    got_t, exp_t = (np.where(k[other] >= 0, x[other], np.inf).astype(np.float64) for k, x in ((prim, t), (want, want_t)))
    nearer = v[np.where(got_t < exp_t, prim[other], want[other])].astype(np.float64)
    for k in range(len(other)):
        if np.isfinite(got_t[k]) and np.isfinite(exp_t[k]) and abs(got_t[k] - exp_t[k]) <= slack[k]:
            continue
        ray = d[other[k]].astype(np.float64)
        corners = nearer[k] - o[other[k]]
        edges = np.roll(corners, -1, 0) - corners
        # distance of the ray's line from each edge's line
        normal = np.cross(edges, ray)
        gap = np.abs((corners * normal).sum(1)) / np.linalg.norm(normal, axis=1)
        assert gap.min() <= slack[k]


@pytest.mark.parametrize("n", [32_768, 32_769, 1_048_576, 2_097_153, 34_000_001])
@pytest.mark.parametrize("bits", [8, 30])
def test_radix_sort_across_scan_tiles(native_library, cuda_device, n, bits):
    """Pair counts at which the digit histogram fills exactly one scan tile,
    one more block, the static scratch's limit, and more tiles than the scan
    of the tile totals takes in one pass: equal to a stable library sort."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda", dtype=torch.int64)
    keys[::3] &= 0xFF   # many equal keys
    k, v = keys.to(torch.int32), torch.arange(n, dtype=torch.int32, device="cuda")
    want, order = torch.sort(keys, stable=True)
    with CudaWavefrontRenderer() as r:
        torch.cuda.synchronize()
        _native.check(r._lib, r._ctx, r._lib.olc_radix_sort_pairs(r._ctx, n, bits, _native.ptr(k), _native.ptr(v)))
        assert torch.equal(k.long(), want)
        assert torch.equal(v.long(), order)


@pytest.mark.parametrize("volumes,step,density", [(1, 0.4, 0.8), (1, 0.05, 60.0), (3, 0.031, 0.5), (8, 0.07, 0.3)])
def test_volume_march_lane_groups(native_library, cuda_device, volumes, step, density):
    """Marches of fewer steps than a ray's lanes, of step counts that are no
    multiple of them, through media so dense that the transmittance ends the
    march inside a group, and through as many overlapping volumes as a scene
    takes: one camera segment per pixel against the oracle's float64 march."""
    import parity_scenes
    from oracle import reference_path_tracer as ref
    from oracle import reference_volume
    from ordinarylight_b200 import scenes

    scene, camera = scenes.box_room()
    tf = ol.Texture1D(np.array([[0.0, 0.0, 0.0, 0.0], [1.0, 0.5, 0.2, 0.3], [0.4, 0.6, 1.0, 0.9]], np.float32))
    for k in range(volumes):
        mat = ol.VolumeMaterial(transfer_function=tf, density_scale=density, emission_scale=0.5, step_size=step,
                                scattering_scale=float(k % 2), scattering_orders=2)
        scene.add_volume(parity_scenes._fbm_field(10 + k, 30 + k) + 0.05, mat,
                         transform=ol.Transform.translation((-0.8 + 0.1 * k, 0.1 + 0.05 * k, -0.7)))
    scene.add_light(ol.PointLight(position=(0.0, 1.7, -0.4), color=(1.0, 0.9, 0.7), intensity=2.0))
    w, h = 23, 17
    with CudaWavefrontRenderer(mode="reference_compatible", max_bounces=1) as r:
        img = r.render_frame(scene, camera, w, h, samples=1)
        o, d = r.camera_rays(camera, w, h, sample=0, frame_index=0)
    tris, _colors, emissions = scene.triangles()
    t, tri = ref.intersect(o.astype(np.float32), d.astype(np.float32), tris)
    vols = scene.visible_volumes
    entries, exits = reference_volume.intersect_unit_boxes(o, d, vols)
    vol_rad, vol_t = reference_volume.integrate_volumes(vols, o, d, entries, exits, max_distance=t, lights=scene.lights)
    surface = np.where((tri >= 0)[:, None], emissions[np.maximum(tri, 0)], ref.sky(d, scene.environment))
    # float32 sums of at most 4,096 steps and an exit at transmittance 1e-4, as the ray-by-ray parity test
    np.testing.assert_allclose(img[..., :3].reshape(-1, 3), vol_rad + vol_t[:, None] * surface, rtol=2e-3, atol=5e-5)


def test_volume_march_lanes_take_several_rays(native_library, cuda_device):
    """More rays (96,000) than a full grid has lane groups (148 SMs x 12
    blocks x 16), so every group marches several, which cross different ones
    of eight scattered volumes: a group's intervals and sources of one ray
    must not reach the next.  600 pixels against the oracle's float64 march."""
    import parity_scenes
    from oracle import reference_path_tracer as ref
    from oracle import reference_volume
    from ordinarylight_b200 import scenes

    scene, camera = scenes.box_room()
    tf = ol.Texture1D(np.array([[0.0, 0.0, 0.0, 0.0], [1.0, 0.5, 0.2, 0.3], [0.4, 0.6, 1.0, 0.9]], np.float32))
    for k in range(8):
        mat = ol.VolumeMaterial(transfer_function=tf, density_scale=0.9, emission_scale=0.3 * k, step_size=0.06,
                                scattering_scale=float(k % 2), scattering_orders=1)
        scene.add_volume(parity_scenes._fbm_field(10 + k, 40 + k) + 0.05, mat,
                         transform=ol.Transform.translation((-0.9 + 0.55 * (k % 4), 0.1 + 0.9 * (k // 4), -0.8 + 0.2 * (k % 3)))
                         @ ol.Transform.scale(0.7))
    scene.add_light(ol.PointLight(position=(0.0, 1.7, -0.4), color=(1.0, 0.9, 0.7), intensity=2.0))
    w, h = 320, 300
    with CudaWavefrontRenderer(mode="reference_compatible", max_bounces=1) as r:
        img = r.render_frame(scene, camera, w, h, samples=1)[..., :3].reshape(-1, 3)
        o, d = r.camera_rays(camera, w, h, sample=0, frame_index=0)
    pick = np.random.default_rng(4).choice(w * h, 600, replace=False)
    o, d = o[pick], d[pick]
    tris, _colors, emissions = scene.triangles()
    t, tri = ref.intersect(o.astype(np.float32), d.astype(np.float32), tris)
    vols = scene.visible_volumes
    entries, exits = reference_volume.intersect_unit_boxes(o, d, vols)
    crossed = (exits > np.maximum(entries, 0.0)).sum(0)
    assert len(set(crossed.tolist())) >= 3      # rays of the picture cross none, one and several of the volumes
    vol_rad, vol_t = reference_volume.integrate_volumes(vols, o, d, entries, exits, max_distance=t, lights=scene.lights)
    surface = np.where((tri >= 0)[:, None], emissions[np.maximum(tri, 0)], ref.sky(d, scene.environment))
    # as the march above: float32 sums and an exit at transmittance 1e-4
    np.testing.assert_allclose(img[pick], vol_rad + vol_t[:, None] * surface, rtol=2e-3, atol=5e-5)


@pytest.mark.parametrize("size", [(1, 1), (1, 5), (2, 2), (7, 3), (64, 64)])
@pytest.mark.parametrize("wrap", ["repeat", "clamp", "mirror"])
@pytest.mark.parametrize("linear", [True, False])
def test_texture_lookups_at_the_wrap_seams(native_library, cuda_device, size, wrap, linear):
    """Coordinates on and one rounding step beside every whole and half
    period, for sizes down to one texel and whole and fractional mip levels,
    against the restated lookup."""
    from oracle import textures as otex
    from ordinarylight_b200.packing import pack_scene

    rng = np.random.default_rng(size[0] * 10 + size[1])
    px = rng.integers(0, 256, (size[1], size[0], 4), dtype=np.uint8)
    scene = ol.Scene()
    quad = np.float32([[-1, 0, -1], [-1, 0, 1], [1, 0, 1], [1, 0, -1]])
    mesh = scene.create_mesh(quad, np.uint32([[0, 1, 2], [0, 2, 3]]),
                             ol.Material(base_color_texture=ol.Texture(px, wrap, wrap, linear)),
                             normals=np.tile(np.float32([0, 1, 0]), (4, 1)), texcoords=quad[:, [0, 2]])
    scene.add_instance(mesh)
    packed = pack_scene(scene)
    marks = np.arange(-4, 5, dtype=np.float32) / 2
    u = np.concatenate([marks, np.nextafter(marks, np.float32(9)), np.nextafter(marks, np.float32(-9)),
                        rng.uniform(-3, 3, 200).astype(np.float32)])
    uv = np.stack(np.meshgrid(u, u), -1).reshape(-1, 2).astype(np.float32)
    fp = rng.choice(np.float32([0.0, 1.0 / max(size), 2.0 / max(size), 0.3, 5.0]), len(uv))
    with CudaWavefrontRenderer() as r:
        for srgb in (False, True):
            got = r.sample_texture(scene, 0, uv, uv, fp, fp, srgb=srgb)
            want = otex.sample_material_texture(packed.texture_words, packed.texture_bindings, 0, uv, uv, srgb, fp, fp)
            # float32 blends (the device may fuse them); a texel coordinate that rounds across a texel's edge
            # moves a nearest lookup to its neighbour, on under 1 in 1,000 of these points
            off = np.abs(got - want).max(1) > 1e-5
            assert off.mean() < (1e-6 if linear else 1e-3)


@pytest.mark.parametrize("triangles", [65, 66, 67, 131_072, 131_073])
@pytest.mark.parametrize("layout", ["soup", "twins", "line"])
def test_planned_collapse_keeps_every_triangle(native_library, cuda_device, triangles, layout):
    """BVH4 nodes and two-triangle leaves planned by the host's and the device's
    builder (up to and above 131,072 triangles), with odd counts, coincident
    triangles (every hit a tie between two) and boxes of zero area: the tree
    validates and hits are the oracle's; visibility agrees with them."""
    from oracle import production

    rng = np.random.default_rng(triangles)
    n = triangles
    if layout == "line":      # triangles in the plane z = 0, in a row: flat boxes
        c = np.zeros((n, 3))
        c[:, 0] = np.arange(n)
        v = c[:, None, :] + np.array([[0.0, 0.0, 0.0], [0.75, 0.0, 0.0], [0.0, 0.75, 0.0]])
    else:
        c = rng.uniform(-20.0, 20.0, (n, 3))
        v = c[:, None, :] + rng.uniform(-0.4, 0.4, (n, 3, 3)) * (8.0 if n < 100 else 1.0)
        if layout == "twins":
            v[1::2] = v[0:n - 1:2][:len(v[1::2])]
    v = v.astype(np.float32)
    scene = _mesh_scene(v.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3))
    rays = 4000
    aim = rng.integers(0, n, rays)
    target = (v[aim].astype(np.float64) * rng.dirichlet((2, 2, 2), rays)[:, :, None]).sum(1)
    away = rng.normal(size=(rays, 3))
    away[:, 2] += np.copysign(0.5, away[:, 2])
    o = (target + 3.0 * away).astype(np.float32)
    d = target - o
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    with CudaWavefrontRenderer() as r:
        assert r.validate_bvh(scene) == 0
        _inst, prim, t, _ = r.trace_closest(scene, o, d, t_min=1e-4)
        hit = prim >= 0
        far = np.where(hit, t * np.float32(1.001) + np.float32(1e-3), np.float32(1e9)).astype(np.float32)
        seen = r.trace_occluded(scene, o, d, far)
        np.testing.assert_array_equal(seen, hit)
    want, want_t = production.trace(scene, o, d, t_min=1e-4)
    assert hit.mean() > 0.9
    # the same triangle (either of two coincident ones from the oracle), or one at the same distance within rounding
    same = (prim >> 1 == want >> 1) if layout == "twins" else (prim == want)
    gap = np.abs(np.where(hit, t, 0.0) - np.where(want >= 0, want_t, 0.0))
    assert np.all(same | (hit & (want >= 0) & (gap <= 4e-6 * np.abs(np.where(hit, t, 1.0)))))
    assert same.mean() > 0.995
    if layout == "twins":     # of two coincident triangles the lower index is reported
        assert np.all(prim[hit & (prim < n - n % 2)] % 2 == 0)
