"""The compressed wide BVH against the BVH2s it is made from, on the CPU.

A host build of the construction and traversal code (tests/wide_bvh_host.cpp)
traces every ray twice, through the wide nodes and through the BVH2s, and the
hits (distance, barycentrics, primitive, instance) and occlusion answers must
agree bit for bit.  The rays are those where the two could part: axis-parallel
ones with zero and denormal components, origins on box planes, through shared
vertices and edges, grazing, from far away and from inside, with directions of
other lengths than 1; the scenes flat, degenerate, duplicated, tiny, huge,
scaled instances, instances and spheres that touch one another, and past the
range the wide test covers."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import acceleration_cases, acceleration_rays
from wfpt import abi, scenes
from wfpt.native import Scene, material

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "wavefront-path-tracer_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    compiler = shutil.which("g++")
    if compiler is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    out = tmp_path_factory.mktemp("wide") / "libwide.so"
    subprocess.run([compiler, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-pthread", "-w",
                    f"-I{CSRC}", f"-I{CUDA_INCLUDE}", "-o", str(out), str(ROOT / "tests" / "wide_bvh_host.cpp"),
                    str(CSRC / "wf_scene.cpp"), str(CSRC / "bvh_build.cpp")], check=True)
    lib = C.CDLL(str(out))

    def run(scene, rays, limits=None):
        rays = np.ascontiguousarray(rays, abi.RAY_DTYPE)
        if limits is None:
            limits = np.random.default_rng(3).uniform(0.1, 20.0, len(rays))
        limits = np.ascontiguousarray(limits, np.float32)
        desc, keep = scene.desc()
        counts = np.zeros(11, np.uint64)
        status = lib.wide_check(C.byref(desc), C.c_void_p(rays.ctypes.data), C.c_void_p(limits.ctypes.data),
                                C.c_uint32(len(rays)), C.c_void_p(counts.ctypes.data))
        assert status == 0
        names = ("closest", "any", "rays", "nodes", "wide_visits", "binary_visits", "usable", "redone", "hits", "tests",
                 "binary_tests")
        got = dict(zip(names, (int(v) for v in counts)))
        assert got["closest"] == 0 and got["any"] == 0, got
        return got
    return run


def make_rays(origins, directions):
    rays = np.zeros(len(origins), abi.RAY_DTYPE)
    rays["origin"], rays["direction"] = origins, directions
    return rays


def hard_rays(points, extent, seed, count=6000):
    """Rays among and at the given points (vertices of the scene): zero and
    denormal components, origins on the points' planes, exact aims at them."""
    rng = np.random.default_rng(seed)
    p = points[rng.integers(0, len(points), count)].astype(np.float32)
    o = rng.uniform(-1.5, 1.5, (count, 3)).astype(np.float32) * np.float32(extent)
    d = rng.normal(0, 1, (count, 3)).astype(np.float32)
    kind = rng.integers(0, 8, count)
    aim = kind <= 2
    d[aim] = p[aim] - o[aim]                                 # through a vertex, any length
    on = kind == 3
    axis = rng.integers(0, 3, count)
    d[on] = 0.0
    d[on, axis[on]] = np.where(rng.random(on.sum()) < 0.5, 1.0, -1.0)
    o[on] = np.where(np.arange(3)[None] == axis[on][:, None], o[on], p[on])  # axis-parallel through a vertex
    zero = kind == 4
    d[zero, axis[zero]] = 0.0                                # in an axis plane, from a vertex's plane
    o[zero, axis[zero]] = p[zero, axis[zero]]
    tiny = kind == 5
    d[tiny, axis[tiny]] = rng.choice([1e-40, -1e-40, 1e-30, -0.0, 1e-12], tiny.sum())
    start = kind == 6
    o[start] = p[start]                                      # from a vertex
    d[np.abs(d).max(1) == 0] = (0, 0, 1)
    return make_rays(o, d)


def soup(n, seed, flat=False, size=0.2):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    v = (c + rng.normal(0, size, (n, 3, 3))).astype(np.float32)
    if flat:
        v[: n // 2, :, 1] = np.round(v[: n // 2, :1, 1] * 4) / 4   # axis-aligned triangles on few planes
    v[::17, 2] = v[::17, 1]                                       # degenerate
    v[1::13] = v[0]                                               # duplicates
    return v


def mesh_scene(v, *instances):
    s = Scene()
    m = s.add_material(material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
    s.add_mesh(scenes.triangles(v[:, 0], v[:, 1], v[:, 2], m))
    s.instances = np.concatenate(instances) if instances else scenes.instance(0)
    return s


@pytest.mark.parametrize("name", list(acceleration_cases()))
def test_acceleration_cases(check, name):
    check(acceleration_cases()[name], acceleration_rays(count=4096))


@pytest.mark.parametrize("count", [1, 2, 3, 4, 7, 8, 9, 24, 25, 200, 3000])
@pytest.mark.parametrize("flat", [False, True])
def test_triangle_soups(check, count, flat):
    v = soup(count, count, flat)
    got = check(mesh_scene(v), hard_rays(v.reshape(-1, 3), 1.0, count))
    assert got["usable"] == 1


def test_grid_of_shared_edges(check):
    """A flat and a bumpy grid: rays at vertices and along edges meet several
    triangles at one distance, which the BVH2s decide."""
    n = 24
    x, z = np.meshgrid(np.linspace(-1, 1, n + 1), np.linspace(-1, 1, n + 1), indexing="ij")
    for bump in (0.0, 0.2):
        p = np.stack([x, bump * np.sin(3 * x) * np.cos(2 * z), z], -1).astype(np.float32)
        a, b, c, d = p[:-1, :-1], p[:-1, 1:], p[1:, 1:], p[1:, :-1]
        v = np.concatenate([np.stack([a, b, c], 2).reshape(-1, 3, 3), np.stack([a, c, d], 2).reshape(-1, 3, 3)])
        got = check(mesh_scene(v), hard_rays(v.reshape(-1, 3), 1.0, 5, 20000))
        assert got["redone"] > 100


@pytest.mark.parametrize("scale,offset", [(1e-9, 0.0), (1e-4, 0.0), (1e3, 0.0), (1.0, 3e4), (1e-3, 1e3), (1e6, 0.0)])
def test_scales_and_offsets(check, scale, offset):
    v = (soup(800, 4, flat=True).astype(np.float64) * scale + offset).astype(np.float32)
    rays = hard_rays(soup(800, 4, flat=True).reshape(-1, 3), 1.0, 6)
    rays["origin"] = rays["origin"] * np.float32(scale) + np.float32(offset)
    got = check(mesh_scene(v), rays, np.random.default_rng(1).uniform(0, 3 * scale, len(rays)))
    assert got["usable"] == 1 and (got["hits"] > 0 or scale < 1e-6)  # hits start at t = 1e-6


@pytest.mark.parametrize("length", [1e-30, 1e-7, 1e-3, 1e3, 1e7, 1e30])
def test_direction_lengths_and_far_origins(check, length):
    v = soup(500, 8)
    rays = hard_rays(v.reshape(-1, 3), 1.0, 9)
    rays["direction"] *= np.float32(length)
    check(mesh_scene(v), rays)
    far = hard_rays(v.reshape(-1, 3), 1.0, 10)
    far["origin"] -= far["direction"] * np.float32(1e5)
    check(mesh_scene(v), far)


@pytest.mark.parametrize("scale,usable", [(1e7, 1), (4e8, 1), (6e8, 1), (2e9, 0)])
def test_large_coordinates(check, scale, usable):
    """Coordinates up to 1e9 (the soup's reach 1.6 times the scale), rays with
    zero and denormal components among them, from within and from far away,
    with short and long directions."""
    v = soup(800, 4, flat=True) / np.float32(1.7)
    s = mesh_scene((v * np.float32(scale)).astype(np.float32),
                   scenes.instance(0), scenes.instance(0, (0.1 * scale, 0, 0), 0.5, 30.0))
    for length in (1.0, 1e-4, 1e4):
        rays = hard_rays(v.reshape(-1, 3), 1.0, 6)
        rays["origin"] *= np.float32(0.6 * scale)
        rays["direction"] *= np.float32(length)
        got = check(s, rays, np.random.default_rng(1).uniform(0, 3 * scale / length, len(rays)))
        assert got["usable"] == usable and (got["hits"] > 0) and (not usable or got["redone"] < len(rays) // 2)


def test_boxes_past_the_range_and_odd_rays(check):
    v = soup(300, 11)
    assert check(mesh_scene(v * np.float32(1e9)), hard_rays(v.reshape(-1, 3) * 1e9, 1e9, 1))["usable"] == 0
    rays = hard_rays(v.reshape(-1, 3), 1.0, 12, 64)
    rays["direction"][0] = (0, 0, 0)
    rays["direction"][1] = (np.nan, 0, 1)
    rays["direction"][2] = (np.inf, 0, 1)
    rays["origin"][3] = (np.nan, 0, 0)
    rays["origin"][4] = (0, np.inf, 0)
    check(mesh_scene(v), rays)


def test_instances_spheres_and_direct_lists(check):
    rng = np.random.default_rng(2)
    v = soup(400, 13, flat=True)
    inst = [scenes.instance(0, rng.uniform(-4, 4, 3), s, 360 * rng.random())
            for s in (1e-7, 1e-3, 0.3, 1.0, 1.0, 2.0, 7.0)] + [scenes.instance(0), scenes.instance(0)]
    s = mesh_scene(v, *inst)
    sp = np.zeros(60, abi.SPHERE_DTYPE)
    sp["center"], sp["radius"] = rng.uniform(-4, 4, (60, 3)), rng.uniform(0.05, 0.8, 60)
    sp["accel"] = np.where(np.arange(60) % 9 == 0, abi.ACCEL_DIRECT, abi.ACCEL_BVH)
    sp[40:50] = sp[10:20]                                         # coincident spheres
    s.spheres = sp
    w = soup(30, 14)
    s.static_triangles = scenes.triangles(w[:, 0], w[:, 1], w[:, 2], 0)
    s.triangles = scenes.triangles(w[:, 0] + 1, w[:, 1] + 1, w[:, 2] + 1, 0)
    got = check(s, hard_rays(np.concatenate([v.reshape(-1, 3), sp["center"]]), 4.0, 15, 20000))
    assert got["redone"] > 0
    only = Scene()
    only.add_material(material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
    only.triangles = scenes.triangles(v[:, 0], v[:, 1], v[:, 2], 0)  # the direct list's own BVH
    check(only, hard_rays(v.reshape(-1, 3), 1.0, 16, 8000))


def unit(d):
    return (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def touching_scene(offset, floor_yaw=0.0, box_yaw=0.0, stack=0, scale=20.0, seed=0):
    """Unit cubes that stand on a scaled cube (its top is y = 0 before the
    offset) and on one another, every one an instance of one mesh."""
    rng = np.random.default_rng(seed)
    s = Scene()
    s.add_material(material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
    s.add_mesh(scenes.box((0, 0, 0), (1, 1, 1), 0, 0))
    inst = [scenes.instance(0, np.add(offset, (0, -scale / 2, 0)), scale, floor_yaw)]
    for _ in range(40):
        x, z = rng.uniform(-0.4 * scale, 0.4 * scale, 2)
        inst.append(scenes.instance(0, np.add(offset, (x, 0.5, z)), 1.0, box_yaw * rng.random()))
        for k in range(stack):
            x, z = x + 0.2 * rng.normal(), z + 0.2 * rng.normal()
            inst.append(scenes.instance(0, np.add(offset, (x, 1.5 + k, z)), 1.0, box_yaw * rng.random()))
    s.instances = np.concatenate(inst)
    return s


@pytest.mark.parametrize("offset", [(0, 0, 0), (100, 3, -50), (1e4, 1e3, -3e3)])
@pytest.mark.parametrize("floor_yaw,box_yaw,stack", [(0.0, 0.0, 0), (0.0, 90.0, 2), (30.0, 90.0, 0)])
def test_touching_instances(check, offset, floor_yaw, box_yaw, stack):
    """Faces that share a plane with other instances' boxes: there the TLAS
    leaf's entry (world ray) and the hit's distance (local ray) round apart,
    and the BVH2's culling order decides.  Rays start within 5 cm of the
    contact plane, as bounces near a contact do, some of them grazing it."""
    s = touching_scene(offset, floor_yaw, box_yaw, stack)
    rng = np.random.default_rng(7)
    n = 100_000
    o = rng.uniform(-9, 9, (n, 3))
    o[:, 1] = rng.uniform(0, 0.05, n) + rng.integers(0, stack + 1, n)
    d = rng.normal(0, 1, (n, 3))
    d[::3, 1] *= 10.0 ** rng.uniform(-3, 0, len(d[::3]))
    got = check(s, make_rays(o + offset, unit(d)))
    assert got["usable"] == 1 and got["hits"] > n // 3


@pytest.mark.parametrize("rise", [0.0, 1e-7, 1e-6, 1e-5, 1e-4, 1e-3])
def test_coincident_surfaces(check, rise):
    """Every instance twice, the copies lifted by `rise`: most hits have
    another at the same distance, which the BVH2s' order decides, or one close
    behind, which it does not."""
    for yaw in (0.0, 90.0):
        s = touching_scene((0, 0, 0), box_yaw=yaw, stack=1)
        copy = s.instances.copy()
        copy["translation"][:, 1] += np.float32(rise)
        s.instances = np.concatenate([s.instances, copy])
        sp = np.zeros(40, abi.SPHERE_DTYPE)
        sp["center"][:20] = np.random.default_rng(1).uniform(-8, 8, (20, 3))
        sp["center"][20:] = sp["center"][:20] + np.float32([0, rise, 0])
        sp["radius"], sp["accel"] = 0.7, abi.ACCEL_BVH
        s.spheres = sp
        rng = np.random.default_rng(8)
        o = rng.uniform(-9, 9, (40_000, 3))
        o[:, 1] = np.abs(o[:, 1]) ** np.where(np.arange(len(o)) % 2 == 0, 1.0, 0.1) - 0.9
        got = check(s, make_rays(o, unit(rng.normal(0, 1, o.shape))))
        # (lifted copies still share the planes of their sides)
        share = got["redone"] / got["hits"]
        assert share > 0.9 if rise == 0.0 else share < (0.5 if rise >= 1e-5 else 1.0)


def test_touching_primitives_of_several_kinds(check):
    """An instance's faces on a static quad's plane, a direct list's and a
    sphere's, and a sphere on the floor instance."""
    for kind in ("static", "list", "sphere", "direct sphere"):
        s = touching_scene((0, 0, 0), box_yaw=45.0)
        floor = scenes.quad((-9, 0, 9), (9, 0, 9), (9, 0, -9), (-9, 0, -9), 0)
        if kind == "static":
            s.static_triangles = floor
        elif kind == "list":
            s.triangles = floor
        else:
            sp = np.zeros(60, abi.SPHERE_DTYPE)
            sp["center"] = np.random.default_rng(1).uniform(-8, 8, (60, 3))
            sp["radius"] = 0.4
            sp["center"][:, 1] = 0.4
            sp["accel"] = abi.ACCEL_BVH if kind == "sphere" else abi.ACCEL_DIRECT
            s.spheres = sp
        rng = np.random.default_rng(8)
        o = rng.uniform(-9, 9, (60_000, 3))
        o[:, 1] = rng.uniform(0, 0.05, len(o))
        check(s, make_rays(o, unit(rng.normal(0, 1, o.shape))))


@pytest.mark.parametrize("radius,ground,near,far", [(0.2, 1000.0, 1e-2, 20.0), (0.2, 1000.0, 20.0, 2e3),
                                                    (0.02, 0.0, 1.0, 1e3), (0.2, 0.0, 1e2, 1e4),
                                                    (5.0, 0.0, 1e-2, 100.0)])
def test_spheres_from_near_and_far(check, radius, ground, near, far):
    """Small spheres that touch, on a large one: from many radii away the
    discriminant cancels and a hit can lie before the sphere's box."""
    rng = np.random.default_rng(3)
    n = 400
    c = rng.uniform(-11, 11, (n, 3))
    c[:, 1] = radius
    turn = rng.uniform(0, 6.3, n // 2)
    c[n // 2:] = c[:n // 2] + 2 * radius * np.stack([np.cos(turn), 0 * turn, np.sin(turn)], 1)
    s = Scene()
    s.add_material(material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
    sp = np.zeros(n + (ground > 0), abi.SPHERE_DTYPE)
    sp["center"][:n], sp["radius"][:n] = c, radius
    if ground:
        sp[n] = ((0, -ground, 0), ground, 0, abi.ACCEL_BVH)
    sp["accel"] = abi.ACCEL_BVH
    s.spheres = sp
    k = 150_000
    at = c[rng.integers(0, n, k)] + radius * unit(rng.normal(0, 1, (k, 3)))
    d = rng.normal(0, 1, (k, 3))
    d[:, 1] = -np.abs(d[:, 1]) * 10.0 ** rng.uniform(-2, 0, k)
    d = unit(d)
    t = np.exp(rng.uniform(np.log(near), np.log(far), (k, 1)))
    check(s, make_rays((at + 0.02 * radius * rng.normal(0, 1, (k, 3)) - d * t).astype(np.float32), d))


@pytest.mark.parametrize("kind,usable", [("sheared", 1), ("strongly sheared", 1), ("not inverse", 0)])
def test_other_instance_transforms(check, kind, usable):
    """Scales after a rotation (|L| |W| of 3, 60 and more than the margins can
    hold), and a world-to-local matrix that is not the other's inverse."""
    s = touching_scene((0, 0, 0), box_yaw=90.0)
    inst = s.instances.copy()
    l2w = inst["local_to_world"].astype(np.float64)
    stretch = {"sheared": 1.5, "strongly sheared": 30.0, "not inverse": 1.0}[kind]
    l2w[1:, :, 0] *= stretch                                # rows of images: scales world x
    inst["local_to_world"] = l2w.astype(np.float32)
    inst["world_to_local"] = np.linalg.inv(l2w).astype(np.float32)
    if kind == "not inverse":
        inst["world_to_local"][3] *= np.float32(1.01)
    s.instances = inst
    rng = np.random.default_rng(9)
    o = rng.uniform(-9, 9, (60_000, 3))
    o[:, 1] = rng.uniform(0, 0.05, len(o))
    assert check(s, make_rays(o, unit(rng.normal(0, 1, o.shape))))["usable"] == usable


def test_scenes_without_bvhs_and_past_the_range_are_traced_once(check):
    """Linear lists alone, and rays or scenes for the BVH2s: no primitive is
    tested twice."""
    rng = np.random.default_rng(6)
    rays = make_rays(rng.uniform(-2, 2, (2000, 3)).astype(np.float32), unit(rng.normal(0, 1, (2000, 3))))
    s = Scene()
    s.add_material(material(abi.MAT_DIFFUSE, (0.5, 0.5, 0.5)))
    sp = np.zeros(9, abi.SPHERE_DTYPE)
    sp["center"], sp["radius"], sp["accel"] = rng.uniform(-2, 2, (9, 3)), 0.4, abi.ACCEL_DIRECT
    s.spheres = sp
    w = soup(12, 3)
    s.static_triangles = scenes.triangles(w[:, 0], w[:, 1], w[:, 2], 0)
    got = check(s, rays)
    assert got["redone"] == 0 and got["tests"] == got["binary_tests"] == 21 * len(rays)
    mesh = mesh_scene(soup(300, 11))
    mesh.spheres, mesh.static_triangles = sp, s.static_triangles
    short = rays.copy()
    short["direction"] *= np.float32(1e-8)
    got = check(mesh, short)
    assert got["redone"] == len(rays) and got["tests"] == got["binary_tests"]
    huge = mesh_scene(soup(300, 11) * np.float32(1e9))
    huge.spheres = sp
    got = check(huge, rays)
    assert got["usable"] == 0 and got["redone"] == len(rays) and got["tests"] == got["binary_tests"]


def test_repository_scenes(check):
    rng = np.random.default_rng(4)
    for scene, _ in (scenes.cornell_box(64, 64), scenes.textured_room(64, 64),
                     scenes.sphere_field(64, 36, frequency=20),
                     scenes.large_mesh(64, 36, terrain_quads=64, instance_count=20, instance_frequency=10,
                                       glass_spheres=4, env_size=(64, 32))):
        o = rng.uniform(-2, 3, (8000, 3)).astype(np.float32)
        d = rng.normal(0, 1, (8000, 3)).astype(np.float32)
        got = check(scene, make_rays(o, d / np.linalg.norm(d, axis=1, keepdims=True)))
        # the Cornell box's boxes stand on its floor: rays from below meet both
        assert got["redone"] < got["rays"] // 50 and got["wide_visits"] < 0.6 * got["binary_visits"], got
