"""Performance cases of the path tracer, each one call that a user's program makes.

`listed()` holds the cases, `draw(rng)` gives one more of the same ranges,
`prepare` builds what a program holds before the call (device scene, renderer
or batch, rays or parameters on the GPU), `run` makes the call, `work` gives
the bytes and operations a pass cannot do without, `tolerance` what outputs
may differ by, and `exact` the 64-bit answer where there is one.

Families:
  render   Renderer.render_task: the task call of a render job or a viewer
           (clear, sample range, read back the radiance sums)
  rays     wf_trace_closest + wf_trace_any on device buffers: visibility and
           light-probe queries of a host program
  guides   wf_frame_guides into a device buffer: a frame's denoiser guides
  batch    Batch: many uneven jobs in one graph, every framebuffer read back
  inverse  wfpt.diff.render and its gradient: one step of inverse rendering
"""
import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parents[1] / "wavefront-path-tracer_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import wfpt  # noqa: E402
from wfpt import abi, diff, scenes  # noqa: E402

MODES = {"graph": abi.MODE_GRAPH, "persistent": abi.MODE_PERSISTENT, "stream": abi.MODE_STREAM}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a viewer's refresh: one sample of a small frame, the shortest call
        dict(name="cornell_preview", kind="render", scene="cornell", width=256, height=256, depth=8, roulette=3,
             spp=1, wave=1, mode="graph"),
        # the Cornell configuration: all 16 samples of a frame in one wave
        dict(name="cornell_16spp", kind="render", scene="cornell", width=256, height=256, depth=8, roulette=3,
             spp=16, wave=16, mode="graph"),
        # the sphere-field configuration at a quarter of its 64 samples:
        # 484 spheres, a 1.3 M-triangle BLAS instanced three times, glass and
        # metal, deep paths
        dict(name="spheres_720p", kind="render", scene="spheres", detail=256, width=1280, height=720, depth=16,
             roulette=16, spp=16, wave=16, mode="graph"),
        # a progressive render of a mesh scene with the library's defaults:
        # one sample of every pixel per launch, odd frame size, no caustics
        dict(name="mesh_progressive", kind="render", scene="mesh", detail=512, width=959, height=541, depth=12,
             roulette=12, spp=1, wave=1, mode="graph", caustics=0),
        # a render job's task on the large mesh: 2.1 M-triangle terrain, 500
        # instances, HDR sun and sky, photon-mapped caustics, full HD
        dict(name="mesh_1080p", kind="render", scene="mesh", detail=1024, width=1920, height=1080, depth=12,
             roulette=12, spp=8, wave=8, mode="graph", caustics=1),
        # glTF-style textured materials, normal maps and alpha masks
        dict(name="textured_room", kind="render", scene="room", width=960, height=540, depth=8, roulette=4,
             spp=4, wave=4, mode="graph"),
        # the reference's cooperative schedule
        dict(name="mesh_persistent", kind="render", scene="mesh", detail=256, width=960, height=540, depth=12,
             roulette=4, spp=2, wave=1, mode="persistent", caustics=0),
        # light probes inside a closed dome: a small query
        dict(name="rays_dome", kind="rays", scene="dome", detail=48, count=65_537),
        # visibility queries over a large mesh scene: a large, odd batch
        dict(name="rays_mesh", kind="rays", scene="mesh", detail=512, count=3_000_001),
        # denoiser guides of a full-HD frame with the previous camera
        dict(name="guides_1080p", kind="guides", scene="mesh", detail=512, width=1920, height=1080),
        # uneven jobs in one graph (the job-batch configuration's ranges)
        dict(name="batch_jobs", kind="batch", jobs=8, size=256, spp=16, depth=8),
        # one inverse-rendering step: image and gradients of 41 k parameters
        dict(name="inverse_step", kind="inverse", cells=32, width=256, height=256, depth=6, spp=8),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "rays", "rays", "guides", "inverse"])
    if kind == "rays":
        scene = rng.choice(["dome", "mesh"])
        detail = _log(rng, 24, 64) if scene == "dome" else _log(rng, 64, 400)
        return dict(kind=kind, scene=scene, detail=detail, count=_log(rng, 1_000, 3_000_000))
    if kind == "guides":
        width = _log(rng, 160, 1920)
        return dict(kind=kind, scene="mesh", detail=_log(rng, 64, 400), width=width, height=max(1, width * 9 // 16))
    if kind == "inverse":
        size = _log(rng, 64, 256)
        return dict(kind=kind, cells=_log(rng, 8, 32), width=size, height=size + rng.randrange(-16, 17),
                    depth=rng.randrange(3, 7), spp=rng.choice([1, 4, 8]))
    scene = rng.choice(["cornell", "spheres", "mesh", "mesh", "room"])
    mode = rng.choice(["graph", "graph", "graph", "stream", "persistent"])
    width = _log(rng, 128, 1280)
    case = dict(kind=kind, scene=scene, width=width, height=max(1, int(width * rng.uniform(0.5, 1.0))),
                depth=rng.randrange(4, 17), roulette=rng.choice([2, 4, 16]), spp=rng.choice([1, 2, 3, 4, 8]), mode=mode)
    case["wave"] = rng.choice([1, case["spp"], case["spp"]]) if mode == "graph" else 1
    if scene == "spheres":
        case["detail"] = _log(rng, 24, 160)
    if scene == "mesh":
        case["detail"] = _log(rng, 64, 400)
        case["caustics"] = rng.choice([0, 1])
    return case


# ---------------------------------------------------------------- preparing
def _dome(detail, seed):
    """A closed bumpy dome of 2 detail^2 triangles (less the poles) around 24
    spheres, as host arrays."""
    rng = np.random.default_rng(seed)
    theta = np.linspace(0.0, math.pi, detail + 1)[:, None]
    phi = np.linspace(0.0, 2.0 * math.pi, detail + 1)[None, :]
    a, b = rng.integers(2, 6, 2)
    r = 10.0 + 0.6 * np.sin(a * phi + rng.uniform(0, 6)) * np.sin(theta) ** 2 + 0.4 * np.sin(b * theta)
    p = np.stack([r * np.sin(theta) * np.cos(phi), r * np.cos(theta) * np.ones_like(phi),
                  r * np.sin(theta) * np.sin(phi)], -1).astype(np.float32)
    p[:, -1] = p[:, 0]
    p[0], p[-1] = p[0, 0], p[-1, 0]
    q = [p[:-1, :-1], p[:-1, 1:], p[1:, 1:], p[1:, :-1]]
    tri = np.concatenate([np.stack([q[0], q[1], q[2]], 2)[1:].reshape(-1, 3, 3),
                          np.stack([q[0], q[2], q[3]], 2)[:-1].reshape(-1, 3, 3)])
    balls = np.zeros((24, 4), np.float32)
    balls[:, :3] = rng.uniform(-6.0, 6.0, (24, 3))
    balls[:, 3] = rng.uniform(0.3, 0.9, 24)
    return tri, balls


def _dome_rays(count, seed):
    """Unit rays from the middle of the dome, made on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    o = torch.rand(count, 3, device="cuda", generator=g) * 10.0 - 5.0
    d = torch.randn(count, 3, device="cuda", generator=g)
    d = d / d.norm(dim=1, keepdim=True)
    limit = torch.rand(count, device="cuda", generator=g) * 14.0 + 1.0
    return torch.cat([o, d], 1).contiguous(), limit


def _scene(case, seed):
    """(host scene, camera) of a case."""
    width, height = case.get("width", 256), case.get("height", 256)
    which = case["scene"]
    if which == "cornell":
        return scenes.cornell_box(width, height)
    if which == "room":
        return scenes.textured_room(width, height)
    if which == "spheres":
        return scenes.sphere_field(width, height, frequency=case["detail"], seed=1 + seed % 10_000)
    if which == "mesh":
        # instance count and their detail follow the terrain's, as in the
        # large-mesh configurations (50 of 18 k triangles to 500 of 200 k)
        detail = case["detail"]
        return scenes.large_mesh(width, height, terrain_quads=detail, instance_count=min(500, 50 + detail // 2),
                                 instance_frequency=min(100, 20 + detail // 8), glass_spheres=20,
                                 env_size=(1024, 512), seed=1 + seed % 10_000)
    tri, balls = _dome(case["detail"], seed)
    s = wfpt.Scene()
    grey = s.add_material(wfpt.material(abi.MAT_DIFFUSE, (0.6, 0.6, 0.6)))
    s.add_mesh(scenes.triangles(tri[:, 0], tri[:, 1], tri[:, 2], grey))
    s.instances = scenes.instance(0)
    sp = np.zeros(len(balls), abi.SPHERE_DTYPE)
    sp["center"], sp["radius"], sp["material"] = balls[:, :3], balls[:, 3], grey
    s.spheres = sp
    s.black_background = True
    return s, None


def _config(case):
    fields = dict(max_depth=case["depth"], rr_start_depth=case.get("roulette", case["depth"]), mode=MODES[case["mode"]])
    if case["mode"] == "graph":
        fields["samples_per_wave"] = case["wave"]
    if case.get("caustics"):
        fields.update(caustics=1, photon_count=500_000)
    return wfpt.render_config(case["width"], case["height"], **fields)


def _batch_sizes(case, k):
    """Resolution, samples and mesh frequency of job k: uneven, each job's own."""
    return max(32, case["size"] >> (k % 3)), max(1, case["spp"] >> (2 * (k % 2))), 16 + 16 * (k % 5)


def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind == "render":
        scene, camera = _scene(case, seed)
        device = wfpt.DeviceScene(scene)
        return dict(kind=kind, case=case, device=device, start=(seed * 64) % 1_000_000,
                    renderer=wfpt.Renderer(device, camera, _config(case)))
    if kind == "rays":
        scene, _ = _scene(case, seed)
        n = case["count"]
        if case["scene"] == "dome":
            rays, limit = _dome_rays(n, seed)
        else:  # points above the terrain, all directions
            g = torch.Generator(device="cuda").manual_seed(seed)
            o = torch.rand(n, 3, device="cuda", generator=g)
            o = o * torch.tensor([100.0, 10.0, 100.0], device="cuda") + torch.tensor([-50.0, 2.0, -50.0], device="cuda")
            d = torch.randn(n, 3, device="cuda", generator=g)
            rays = torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).contiguous()
            limit = torch.rand(n, device="cuda", generator=g) * 60.0 + 1.0
        return dict(kind=kind, device=wfpt.DeviceScene(scene), rays=rays, limit=limit, count=n,
                    hits=torch.empty(n * 17, dtype=torch.float32, device="cuda"),
                    occluded=torch.empty(n, dtype=torch.uint8, device="cuda"))
    if kind == "guides":
        scene, camera = _scene(case, seed)
        previous = scenes.look_at_camera((0.2, 14.0, 38.2), (0.0, 0.0, 0.0), 50.0, case["width"], case["height"])
        return dict(kind=kind, case=case, device=wfpt.DeviceScene(scene), camera=camera, previous=previous,
                    out=torch.empty(case["width"] * case["height"] * 14, dtype=torch.float32, device="cuda"))
    if kind == "batch":
        jobs = []
        for k in range(case["jobs"]):
            size, spp, frequency = _batch_sizes(case, k)
            scene, camera = scenes.sphere_field(size, size, frequency=frequency, seed=1 + (seed * 31 + k) % 10_000)
            jobs.append(dict(scene=wfpt.DeviceScene(scene), camera=camera, sample_start=(seed * 64) % 1_000_000,
                             config=wfpt.render_config(size, size, max_depth=case["depth"]), sample_count=spp))
        return dict(kind=kind, jobs=jobs, batch=wfpt.Batch(jobs))
    scene, camera, n, _ = scenes.cornell_inverse(case["width"], case["height"], cells=case["cells"])
    albedo, rough = scenes.inverse_parameters(scene, n, seed=100 + seed % 10_000)
    g = torch.Generator(device="cuda").manual_seed(seed)
    config = diff.diff_config(case["width"], case["height"], case["spp"], case["depth"], n,
                              sample_start=(seed * 64) % 1_000_000)
    return dict(kind=kind, device=wfpt.DeviceScene(scene), camera=camera, config=config,
                albedo=torch.from_numpy(albedo).cuda().requires_grad_(True),
                rough=torch.from_numpy(rough).cuda().requires_grad_(True),
                scale=torch.tensor([1.0 + 0.1 * (seed % 7)], device="cuda", requires_grad=True),
                adjoint=torch.randn(case["height"], case["width"], 3, device="cuda", generator=g))


# ------------------------------------------------------------------ running
def run(state):
    kind = state["kind"]
    if kind == "render":
        c = state["case"]
        return state["renderer"].render_task((0, 0, c["width"], c["height"]), state["start"], c["spp"])
    if kind == "rays":
        lib, scene, n = wfpt.library(), state["device"].handle, state["count"]
        rays, hits, occluded = state["rays"], state["hits"], state["occluded"]
        stream = torch.cuda.current_stream().cuda_stream
        wfpt.check(lib.wf_trace_closest(scene, rays.data_ptr(), n, hits.data_ptr(), stream))
        wfpt.check(lib.wf_trace_any(scene, rays.data_ptr(), state["limit"].data_ptr(), n, occluded.data_ptr(), stream))
        rows = hits.view(n, 17)  # t, position, geometric normal, normal | five ids | u, v
        return dict(t=rows[:, 0], position=rows[:, 1:4], geometric_normal=rows[:, 4:7], normal=rows[:, 7:10],
                    ids=hits.view(torch.int32).view(n, 17)[:, 10:15], uv=rows[:, 15:17], occluded=occluded)
    if kind == "guides":
        c, out = state["case"], state["out"]
        now, before = wfpt.camera_struct(state["camera"]), wfpt.camera_struct(state["previous"])
        wfpt.check(wfpt.library().wf_frame_guides(
            state["device"].handle, C.byref(now), C.byref(before), c["width"], c["height"], 0, 0, c["width"],
            c["height"], out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return out.view(torch.int32).view(c["height"], c["width"], 14)  # the 56-byte records, bit for bit
    if kind == "batch":
        batch = state["batch"]
        batch.reset()
        batch.run()
        return [batch.download(k) for k in range(len(state["jobs"]))]
    parameters = (state["albedo"], state["rough"], state["scale"])
    image = diff.render(state["device"], state["camera"], state["config"], *parameters)
    return [image] + list(torch.autograd.grad(image, parameters, state["adjoint"]))


# --------------------------------------------------------------------- work
def _triangles(case):
    """Triangles a case's scene holds in memory."""
    which = case.get("scene")
    if which == "spheres":
        return 20 * case["detail"] ** 2
    if which == "mesh":
        return 2 * case["detail"] ** 2 + 20 * min(100, 20 + case["detail"] // 8) ** 2
    if which == "dome":
        return 2 * case["detail"] ** 2
    return {"cornell": 36, "room": 280}.get(which, 10 * case.get("cells", 16) ** 2)


def _ray_flops(triangles):
    """A ray's least work: one descent of a balanced binary tree (two box
    tests of 24 operations per level) and one triangle test (about 60)."""
    return 48.0 * math.log2(max(2, triangles)) + 60.0


def work(case):
    """36 bytes per triangle of the scene read once, inputs and outputs once;
    per path at least one extension ray, one shadow ray and one shading
    evaluation (about 200 operations)."""
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for k in range(case["jobs"]):
            size, spp, frequency = _batch_sizes(case, k)
            triangles = 20 * frequency ** 2
            total["bytes"] += 36.0 * triangles + 12.0 * size * size
            total["flops"] += size * size * spp * (2.0 * _ray_flops(triangles) + 200.0)
        return total
    triangles = _triangles(case)
    per_ray = _ray_flops(triangles)
    if kind == "rays":
        n = case["count"]
        return dict(bytes=36.0 * triangles + n * (24.0 + 68.0 + 24.0 + 4.0 + 1.0), flops=2.0 * n * per_ray)
    pixels = case["width"] * case["height"]
    if kind == "guides":
        return dict(bytes=36.0 * triangles + 56.0 * pixels, flops=2.0 * pixels * per_ray)
    if kind == "inverse":  # the gradient replays the image's paths
        return dict(bytes=2 * (36.0 + 16.0) * triangles + 24.0 * pixels,
                    flops=2.0 * pixels * case["spp"] * (2.0 * per_ray + 200.0))
    return dict(bytes=36.0 * triangles + 12.0 * pixels, flops=pixels * case["spp"] * (2.0 * per_ray + 200.0))


def tolerance(case):
    """Renders, ray queries and guides are bit-exact by contract (the image
    does not depend on schedule or tree), so another correct implementation
    at this precision returns the same bits.  Gradients are float terms added
    by atomics in no fixed order."""
    return {"rel": 1e-5} if case["kind"] == "inverse" else "exact"


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """Closest hits of the dome by testing every triangle and sphere in 64
    bits.  The other cases have no closed answer: their paths depend on random
    streams and on every earlier decision, or would take minutes."""
    if case["kind"] != "rays" or case["scene"] != "dome" or case["count"] > 400_000:
        return None
    tri, balls = _dome(case["detail"], int(seed))
    rays, _ = _dome_rays(case["count"], int(seed))
    tri = torch.from_numpy(tri).cuda().double()
    balls = torch.from_numpy(balls).cuda().double()
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    normal = torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=1)
    position, facing = [], []
    for part in rays.double().split(2048):
        o, d = part[:, None, :3], part[:, None, 3:]
        p = torch.linalg.cross(d.expand(-1, len(tri), -1), e2[None].expand(len(part), -1, -1))
        inv = 1.0 / (e1[None] * p).sum(-1)
        s = o - v0[None]
        u = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        v = (d * q).sum(-1) * inv
        t = (e2[None] * q).sum(-1) * inv
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-6), t, torch.inf)
        t, which = t.min(1)
        oc = o - balls[None, :, :3]
        b = (oc * d).sum(-1)
        a = (d * d).sum(-1)
        disc = b * b - a * ((oc * oc).sum(-1) - balls[None, :, 3] ** 2)
        root = disc.clamp(min=0).sqrt()
        near, far = (-b - root) / a, (-b + root) / a
        ts = torch.where(near > 1e-6, near, far)
        ts = torch.where((disc >= 0) & (ts > 1e-6), ts, torch.inf)
        ts, ball = ts.min(1)
        on_ball = ts < t
        at = part[:, :3] + part[:, 3:] * torch.where(on_ball, ts, t)[:, None]
        n = normal[which]
        n = torch.where((n * part[:, 3:]).sum(1, keepdim=True) > 0, -n, n)
        out = torch.nn.functional.normalize(at - balls[ball, :3], dim=1)
        position.append(at)
        facing.append(torch.where(on_ball[:, None], out, n))
    return dict(t=None, position=torch.cat(position), geometric_normal=torch.cat(facing), normal=None, ids=None,
                uv=None, occluded=None)
