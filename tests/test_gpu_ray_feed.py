"""Launches of every size through the trace and shadow kernels' ray feed.

A launch of few rays uses some lanes of each warp, a larger one all of them
and then refills.  Every path's radiance is independent of the launch it runs
in, so a frame must not change with the number of samples per wave, the
wavefronts per tile or the schedule (bit for bit), from one pixel to more rays
than the launch has lanes."""
import numpy as np
import pytest

import wfpt
from wfpt import abi, scenes

pytestmark = pytest.mark.gpu


def _scene(which, w, h):
    if which == "mesh":
        return scenes.large_mesh(w, h, terrain_quads=48, instance_count=12, instance_frequency=8, glass_spheres=4,
                                 env_size=(64, 32))
    if which == "spheres":  # no lights and no environment: shading without shadow rays
        return scenes.sphere_field(w, h, frequency=8, seed=5)
    if which == "room":  # alpha-masked textures
        return scenes.textured_room(w, h)
    if which == "masked lists":  # both: the fully generic kernels
        scene, cam = scenes.textured_room(w, h)
        lamp = scene.add_material(wfpt.material(abi.MAT_EMISSIVE, (1, 1, 1), (8, 8, 8)))
        scene.material_textures = np.concatenate([scene.material_textures, scenes.material_textures()])
        scene.static_triangles = scenes.quad((-.2, .9, -.2), (.2, .9, -.2), (.2, .9, .2), (-.2, .9, .2), lamp)
        return scene, cam
    if which == "contact":  # glass cubes on an instanced floor, seen from among them: faces on one plane
        scene = wfpt.Scene()
        rng = np.random.default_rng(5)
        mats = [scene.add_material(wfpt.material(t, c, ior=1.5)) for t, c in
                ((abi.MAT_DIFFUSE, (0.6, 0.5, 0.4)), (abi.MAT_DIELECTRIC, (1, 1, 1)), (abi.MAT_DIFFUSE, (0.2, 0.6, 0.3)))]
        scene.add_mesh(scenes.box((0, 0, 0), (1, 1, 1), 0, mats[0]))
        scene.instances = np.concatenate(
            [scenes.instance(0, (0, -10, 0), 20.0)] +
            [scenes.instance(0, (x, 0.5, z), 1.0, 0.0, mats[1 + k % 2])
             for k, (x, z) in enumerate(rng.uniform(-6, 6, (60, 2)))])
        return scene, scenes.look_at_camera((0.494, 0.02, 6.4), (0.45, -0.3, 6.2), 90.0, w, h)
    scene, cam = scenes.cornell_box(w, h)
    if which == "lists":  # primitives outside the BVHs
        scene.static_triangles = scenes.quad((-1, 0, 1), (1, 0, 1), (1, 0.5, 1), (-1, 0.5, 1), 1)
        scene.triangles = scenes.quad((-1, 1, 1), (0, 1, 1), (0, 2, 0.5), (-1, 2, 0.5), 2)
    return scene, cam


@pytest.mark.parametrize("which", ["cornell", "mesh", "spheres", "room", "lists", "masked lists", "contact"])
@pytest.mark.parametrize("size", [(1, 1), (3, 5), (65, 33), (257, 129)])
def test_frame_does_not_depend_on_launch_size(cuda, which, size):
    w, h = size
    scene, cam = _scene(which, w, h)
    dev = wfpt.DeviceScene(scene)
    spp = 8
    images = []
    for fields in (dict(mode=abi.MODE_GRAPH), dict(mode=abi.MODE_GRAPH, samples_per_wave=8),
                   dict(mode=abi.MODE_GRAPH, samples_per_wave=8, concurrent_tiles=1),
                   dict(mode=abi.MODE_STREAM),
                   dict(mode=abi.MODE_PERSISTENT, persistent_stages=abi.PERSISTENT_FUSED),
                   dict(mode=abi.MODE_PERSISTENT, persistent_stages=abi.PERSISTENT_STAGED)):
        r = wfpt.Renderer(dev, cam, wfpt.render_config(w, h, max_depth=8, rr_start_depth=4, **fields))
        images.append(r.render_task((0, 0, w, h), 3, spp))
        r.close()
    dev.close()
    for image in images[1:]:
        assert np.array_equal(images[0].view(np.uint32), image.view(np.uint32))


def test_more_rays_than_lanes(cuda):
    """1.2 M rays per bounce against at most 151,552 lanes."""
    scene, cam = scenes.cornell_box(320, 240)
    dev = wfpt.DeviceScene(scene)
    images = []
    for wave in (1, 16):
        r = wfpt.Renderer(dev, cam, wfpt.render_config(320, 240, max_depth=5, samples_per_wave=wave))
        images.append(r.render_task((0, 0, 320, 240), 0, 16))
        r.close()
    dev.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))


@pytest.mark.parametrize("which", ["mesh", "room", "lists", "masked lists"])
def test_large_ray_batches_match_small_ones(cuda, which):
    """Batches around the size from which lanes are refilled (8 CTAs of 128 on
    each SM, twice) against the same rays in small ones, record for record."""
    scene, _ = _scene(which, 64, 36)
    dev = wfpt.DeviceScene(scene)
    line = cuda.cuda.get_device_properties(0).multi_processor_count * 8 * 256
    rng = np.random.default_rng(2)
    rays = np.zeros(line + 4097, abi.RAY_DTYPE)
    rays["origin"] = rng.uniform(-2, 3, (len(rays), 3))
    d = rng.normal(0, 1, (len(rays), 3))
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["direction"][::1001] *= np.float32(1e-8)  # past the wide test's bounds: the BVH2s decide
    limit = rng.uniform(0.1, 6.0, len(rays)).astype(np.float32)
    part = 50_000
    hits = np.concatenate([dev.trace_closest(rays[k:k + part]) for k in range(0, len(rays), part)])
    occluded = np.concatenate([dev.trace_any(rays[k:k + part], limit[k:k + part]) for k in range(0, len(rays), part)])
    for count in (line - 1, line, line + 1, len(rays)):
        assert dev.trace_closest(rays[:count]).tobytes() == hits[:count].tobytes()
        assert np.array_equal(dev.trace_any(rays[:count], limit[:count]), occluded[:count])
    dev.close()


@pytest.mark.parametrize("lists", [False, True])
@pytest.mark.parametrize("masked", [False, True])
def test_ray_batches_do_not_depend_on_their_route(cuda, lists, masked):
    """Which kernel traces a batch depends on the leaves of the scene's trees
    (32 and 64 of them, 64 in the TLAS) and on its size.  Far and tiny spheres
    that no ray meets change the count and must change nothing else."""
    w, h = 64, 64
    line = cuda.cuda.get_device_properties(0).multi_processor_count * 8 * 256
    rng = np.random.default_rng(3)
    rays = np.zeros(line + 33, abi.RAY_DTYPE)
    rays["origin"] = rng.uniform(-0.9, 0.9, (len(rays), 3))
    d = rng.normal(0, 1, (len(rays), 3))
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    limit = rng.uniform(0.1, 3.0, len(rays)).astype(np.float32)
    answers = []
    for far in (0, 1, 32, 33, 33, 62, 63, 64):
        scene = wfpt.Scene()
        mat = scene.add_material(wfpt.material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
        half = scene.add_material(wfpt.material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
        if masked:
            scene.materials[half]["alpha_masked"] = 1
            scene.materials[half]["opacity"] = 0.0
            scene.textures = [np.full((1, 1, 4), 255, np.uint8)]
            scene.material_textures = scenes.material_textures()
            scene.material_textures = np.concatenate(
                [scene.material_textures, scenes.material_textures(albedo=scenes.texture_binding(0))])
        v = (rng2 := np.random.default_rng(4)).uniform(-1, 1, (30, 1, 3)) + rng2.normal(0, 0.3, (30, 3, 3))
        scene.add_mesh(scenes.triangles(*v.astype(np.float32).transpose(1, 0, 2), np.where(np.arange(30) % 3, mat, half)))
        scene.instances = scenes.instance(0)
        if lists:
            scene.static_triangles = scenes.quad((-1, -0.7, 1), (1, -0.7, 1), (1, -0.7, -1), (-1, -0.7, -1), mat)
        sp = np.zeros(far, abi.SPHERE_DTYPE)
        sp["center"] = 1e6 + np.arange(far)[:, None]
        sp["radius"], sp["material"], sp["accel"] = 1e-3, mat, abi.ACCEL_BVH
        scene.spheres = sp
        dev = wfpt.DeviceScene(scene)
        for count in (1, 33, len(rays)):
            answers.append((count, dev.trace_closest(rays[:count]).tobytes(),
                            dev.trace_any(rays[:count], limit[:count]).tobytes()))
        dev.close()
    want = {count: (hits, occluded) for count, hits, occluded in answers[:3]}
    assert 0 < sum(want[len(rays)][1]) < len(rays)
    for count, hits, occluded in answers:
        assert hits == want[count][0] and occluded == want[count][1]


@pytest.mark.parametrize("capacity,pass_paths", [(0, 0), (33, 0), (300, 1021)])
def test_batch_of_scenes_without_lights(cuda, capacity, pass_paths):
    """A batch of sphere fields shades without shadow rays; its images are
    those of the streaming schedule, which always queues them."""
    jobs, want = [], []
    for w, h, depth, count, seed in ((31, 17, 6, 3, 1), (64, 40, 16, 2, 2), (1, 1, 1, 5, 3)):
        scene, cam = scenes.sphere_field(w, h, frequency=8, seed=seed)
        dev = wfpt.DeviceScene(scene)
        jobs.append(dict(scene=dev, camera=cam, sample_start=7, sample_count=count,
                         config=wfpt.render_config(w, h, max_depth=depth)))
        r = wfpt.Renderer(dev, cam, wfpt.render_config(w, h, max_depth=depth, mode=abi.MODE_STREAM))
        want.append(r.render_task((0, 0, w, h), 7, count))
        r.close()
    batch = wfpt.Batch(jobs, slot_capacity=capacity, pass_paths=pass_paths)
    for _ in range(2):
        batch.reset()
        batch.run()
        batch.synchronize()
        for k, image in enumerate(want):
            assert np.array_equal(batch.download(k).view(np.uint32), image.view(np.uint32))
    batch.close()
    for job in jobs:
        job["scene"].close()


@pytest.mark.parametrize("which,direct", [("spheres", True), ("cornell", False)])
def test_stage_profile_times_the_kernels_of_the_graph(cuda, which, direct):
    """A scene that shades without shadow rays has no shadow and finalize
    launches; the profiled passes add the same samples as the graph."""
    w, h, depth = 65, 33, 6
    scene, cam = _scene(which, w, h)
    dev = wfpt.DeviceScene(scene)
    cfg = wfpt.render_config(w, h, max_depth=depth, rr_start_depth=4)
    r = wfpt.Renderer(dev, cam, cfg)
    p = r.profile_sample()
    assert p["shade"]["launches"] == p["trace"]["launches"] == depth
    assert p["shadow"]["launches"] == p["finalize"]["launches"] == (0 if direct else depth)
    assert p["shadow_rays"] == 0 if direct else p["shadow_rays"] > 0
    plain = wfpt.Renderer(dev, cam, cfg)  # the timed pass and the counting one are samples 0 and 1
    want = plain.render_task((0, 0, w, h), 0, 2)
    assert np.array_equal(r.download().view(np.uint32), want.view(np.uint32))
    r.close()
    plain.close()
    dev.close()


@pytest.mark.parametrize("frequency", [4, 72])  # the builder's scratch under and over a megabyte
def test_scene_creation_does_not_wait_for_other_streams(cuda, frequency):
    """A scene is made while another stream is busy for about a second."""
    torch = cuda
    scene = wfpt.Scene()
    scene.add_mesh(scenes.geodesic_sphere(frequency, scene.add_material(wfpt.material(abi.MAT_DIFFUSE, (1, 1, 1)))))
    scene.instances = scenes.instance(0)
    wfpt.DeviceScene(scene).close()  # loads the kernels
    torch.cuda.synchronize()
    busy = torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)
        end = torch.cuda.Event()
        end.record()
    dev = wfpt.DeviceScene(scene)
    still_busy = not end.query()
    torch.cuda.synchronize()
    dev.close()
    assert still_busy


def test_guides_do_not_depend_on_the_tile(cuda):
    """Pixels go to the warps in blocks for tiles of two resident waves (16
    CTAs of 128 an SM) and more, in rows for smaller ones."""
    line = cuda.cuda.get_device_properties(0).multi_processor_count * 16 * 128
    w, h = 701, line // 701 + 3
    scene, cam = _scene("mesh", w, h)
    dev = wfpt.DeviceScene(scene)
    whole = dev.frame_guides(cam, w, h)
    assert w * h > line and 0 < int((whole["valid"] != 0).sum()) < w * h
    for x, y, tw, th in ((0, 0, w, h // 2), (0, h // 2, 333, h - h // 2), (333, h // 2, w - 333, h - h // 2),
                         (0, 0, w, h - 4), (17, 5, 1, 1), (3, 7, 31, 5)):
        tile = dev.frame_guides(cam, w, h, tile=(x, y, tw, th))
        assert tile.tobytes() == np.ascontiguousarray(whole[y:y + th, x:x + tw]).tobytes()
    dev.close()
