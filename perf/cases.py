"""The work that a user of the ray-tracing core has it do, as cases that can be timed.

Four kinds of pass, all through the package's host classes or the C ABI behind them:

* ``query``: rays against a mesh (a ray buffer on the device, or page-locked host buffers).  With
  ``rebuild`` the pass first rebuilds what changed since the last one, as an animated scene does:
  the TLAS (moving instances) or the BLAS and the TLAS (a deforming mesh).
* ``frame``: one frame of the render loop.  The TLAS is rebuilt, or refitted in place, from the
  frame's instance records, and the frame is traced into its RGBA8 image.
* ``batch``: many scenes of different sizes in one batched launch sequence.
* ``serve``: a burst of render requests to a server over resident scenes.

An acceleration structure's bytes are the library's own affair; what a user gets from a build is
the hits of the rays traced through it, so builds are followed by a query and return its hits.
Loading files (GLB, PNG) happens once when a program starts and is not a case of its own; the
default scene's preparation goes through it.
"""
from __future__ import annotations

import ctypes
import functools
import importlib
import math

import numpy as np
import torch

_PACKAGE = "ray-tracing-gallery_gb300"
abi = importlib.import_module(_PACKAGE + ".abi")
assets = importlib.import_module(_PACKAGE + ".assets")
host = importlib.import_module(_PACKAGE + ".host")
scenes = importlib.import_module(_PACKAGE + ".scenes")

TLAS_FLAGS = abi.RT_BUILD_PREFER_FAST_TRACE | abi.RT_BUILD_ALLOW_UPDATE
FRAME_SCENES = ("small", "gallery", "default", "full")
RESOLUTIONS = ((128, 128), (256, 256), (512, 512), (1024, 1024), (1280, 720), (1920, 1080))
BRUTE_FORCE_PAIRS = 2e10  # ray-triangle pairs that a 64-bit brute-force search does in a few seconds


def _query(name, triangles, instances, rays, rebuild="none", nodes="fp32", prefer="trace", buffers="device"):
    return {"name": name, "kind": "query", "triangles": triangles, "instances": instances, "rays": rays,
            "rebuild": rebuild, "nodes": nodes, "prefer": prefer, "buffers": buffers}


def _frame(name, scene, width, height, update):
    return {"name": name, "kind": "frame", "scene": scene, "width": width, "height": height, "update": update}


def listed():
    return [
        # Picking and line-of-sight tests: a few rays at a time against one small model.
        _query("pick_1k_rays", 4096, 1, 1024),
        # A small deforming model (cloth, a skinned figure) rebuilt every frame for fast builds, then probed.
        _query("rebuild_4k_triangles", 4096, 4, 4096, rebuild="blas", prefer="build"),
        # A mid-size deforming model, rebuilt for fast traces as the reference builds every BLAS.
        _query("rebuild_160k_triangles", 163_840, 1, 16_384, rebuild="blas"),
        # Loading or re-meshing a scan: the largest mesh of the benchmark, built and then probed.
        _query("rebuild_10m_triangles", 10_485_760, 1, 262_144, rebuild="blas"),
        # A crowd: thousands of moving instances, the TLAS rebuilt every frame, an odd number of rays.
        _query("rebuild_10k_instances", 4096, 10_007, 250_001, rebuild="tlas"),
        # The benchmark's precision workload: random rays through the largest mesh, FP32 nodes.
        _query("trace_4m_rays", 10_485_760, 1, 4_194_304),
        # Baking or visibility from a host program: page-locked host buffers, quantised nodes, an odd count.
        _query("trace_1m_rays_host", 655_360, 1, 1_000_003, nodes="quantised", buffers="host"),
        # A thumbnail or preview: 17 instances, one hard shadow; launches and latency count.
        _frame("frame_256x256", "small", 256, 256, "rebuild"),
        # The reference's own scene at its own size, refitted every frame: textures, mirrors, a portal, alpha.
        _frame("frame_720p_default", "default", 1280, 720, "refit"),
        # The benchmark's full frame: 256 moving instances, four soft shadows, one bounce.
        _frame("frame_1080p_full", "full", 1920, 1080, "rebuild"),
        # The benchmark's batching form: scenes of many sizes in one launch sequence, quantised, camera-ray packets.
        {"name": "batch_12_scenes", "kind": "batch", "scenes": 12, "triangles": 300_000, "nodes": "quantised",
         "packets": True},
        # The benchmark's serving form: a burst of requests of mixed sizes over resident scenes.
        {"name": "serve_24_requests", "kind": "serve", "scenes": 4, "triangles": 100_000, "requests": 24},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("query", "query", "query", "frame", "frame", "batch", "serve"))
    if kind == "query":
        rebuild = rng.choice(("none", "tlas", "blas"))
        triangles = _log_uniform(rng, 500, 10_000_000)
        instances = 1 if rebuild != "tlas" else _log_uniform(rng, 2, 10_000)
        if rebuild == "tlas":
            triangles = min(triangles, 200_000)
        c = _query("", triangles, instances, _log_uniform(rng, 1000, 4_000_000 if rebuild == "none" else 250_000),
                   rebuild, rng.choice(("fp32", "quantised")), rng.choice(("trace", "trace", "build")),
                   rng.choice(("device", "device", "host")))
        del c["name"]
        return c
    if kind == "frame":
        height = _log_uniform(rng, 90, 1080)
        c = _frame("", rng.choice(FRAME_SCENES), max(96, int(height * rng.uniform(1.0, 16 / 9))), height,
                   rng.choice(("rebuild", "refit")))
        del c["name"]
        return c
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 12), "triangles": _log_uniform(rng, 20_000, 300_000),
                "nodes": rng.choice(("fp32", "quantised")), "packets": rng.random() < 0.5}
    return {"kind": "serve", "scenes": rng.randint(2, 4), "triangles": _log_uniform(rng, 20_000, 100_000),
            "requests": rng.randint(6, 24)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _sphere_grid(triangles):
    """Longitude and latitude cells of a sphere of about `triangles` triangles (two per cell)."""
    nv = max(4, int(round(math.sqrt(triangles / 4.0))))
    return max(4, int(round(triangles / (2.0 * nv)))), nv


def _bumpy_sphere(triangles, rng):
    """A displaced sphere (radius 10) on the device: float32 positions, uint32 indices."""
    nu, nv = _sphere_grid(triangles)
    dev = torch.device("cuda")
    phi = torch.arange(nu + 1, dtype=torch.float64, device=dev)[:, None] * (2 * math.pi / nu)
    theta = torch.arange(nv + 1, dtype=torch.float64, device=dev)[None, :] * (math.pi / nv)
    x, y, z = (torch.sin(theta) * torch.cos(phi), torch.cos(theta) + 0 * phi, torch.sin(theta) * torch.sin(phi))
    r = torch.full_like(x, 10.0)
    for octave in range(6):  # bumps of ever finer detail, as a scan has
        f = rng.normal(size=3) * 2.0 * 2.0 ** octave
        r += 0.5 * 0.5 ** octave * torch.sin(f[0] * x + f[1] * y + f[2] * z + rng.uniform(0.0, 2 * math.pi))
    positions = torch.stack([r * x, r * y, r * z], -1).reshape(-1, 3).to(torch.float32)
    a = (torch.arange(nu, device=dev)[:, None] * (nv + 1) + torch.arange(nv, device=dev)[None, :]).reshape(-1)
    b = a + nv + 1
    cells = torch.stack([a, a + 1, b + 1, a, b + 1, b], -1)
    return positions, cells.reshape(-1, 3).to(torch.int32).contiguous()


def _random_rays(count, box, rng):
    """Origins uniform in a box around the scene, directions uniform on the sphere."""
    rays = np.zeros(count, abi.RAY_DTYPE)
    rays["origin"] = ((rng.random((count, 3), np.float32) - 0.5) * box)
    d = rng.standard_normal((count, 3), np.float32)
    rays["direction"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["tmax"] = np.inf
    return rays


def _rotations(count, rng):
    q = rng.normal(size=(count, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(count, 3, 3)


def _transforms(count, rng):
    """One model where it stands, or many turned and scattered at an even density."""
    m = np.zeros((count, 3, 4), np.float32)
    if count == 1:
        m[0, :, :3] = np.eye(3)
        return m, 30.0
    box = 30.0 * count ** (1 / 3)
    m[:, :, :3] = _rotations(count, rng) * rng.uniform(0.5, 1.5, (count, 1, 1))
    m[:, :, 3] = rng.uniform(-box / 2, box / 2, (count, 3))
    return m, box


def _pinned(a):
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    t.numpy()[:] = a.view(np.uint8).reshape(-1)
    return t


def _query_inputs(case, seed):
    rng = np.random.default_rng(seed)
    positions, indices = _bumpy_sphere(case["triangles"], rng)
    transforms, box = _transforms(case["instances"], rng)
    return positions, indices, transforms, _random_rays(case["rays"], box, rng)


def _prepare_query(case, seed):
    positions, indices, transforms, rays = _query_inputs(case, seed)
    device = host.Device()
    flags = abi.RT_BUILD_PREFER_FAST_TRACE if case["prefer"] == "trace" else abi.RT_BUILD_PREFER_FAST_BUILD
    flags |= abi.RT_BUILD_QUANTIZED_NODES if case["nodes"] == "quantised" else 0
    scratch = host.ScratchBuffer()
    geometry = host.GeometryDesc(positions.data_ptr(), indices.data_ptr(), indices.numel(), len(positions), True)
    blas = host.AccelerationStructure.build_blas(device, "mesh", scratch, [geometry], flags)
    records = scenes.instance_records(transforms, 0, 0, abi.HIT_SHADER_TEXTURED)
    records["blas"] = blas.device_address()
    instances = host.Device.upload(records)
    tlas = host.AccelerationStructure.build_tlas(device, instances, len(records), scratch)
    n = len(rays)
    if case["buffers"] == "host":
        ray_buffer = _pinned(rays)
        hit_buffer = torch.empty(n * abi.HIT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
    else:
        ray_buffer = host.Device.upload(rays)
        hit_buffer = host.Device.alloc(n * abi.HIT_DTYPE.itemsize)
    return {"case": case, "device": device, "mesh": (positions, indices), "geometry": geometry, "scratch": scratch,
            "blas": blas, "instances": instances, "tlas": tlas, "rays": ray_buffer, "hits": hit_buffer, "count": n}


def _run_query(s):
    case, device = s["case"], s["device"]
    if case["rebuild"] == "blas":
        s["blas"].rebuild_blas(device, s["scratch"], [s["geometry"]])
    if case["rebuild"] != "none":
        s["tlas"].rebuild_tlas(device, s["instances"], case["instances"], s["scratch"])
    stream = device.stream_handle()
    if case["buffers"] == "host":
        device.check(device.lib.rt_trace_ray_buffer_host(device.ctx, s["tlas"].device_address(), None, None, 0, 0xFF, 0,
                                                         s["rays"].data_ptr(), s["count"], s["hits"].data_ptr(), 0,
                                                         stream))
        torch.cuda.current_stream().synchronize()  # the caller reads host memory next
    else:
        device.check(device.lib.rt_cmd_trace_ray_buffer(device.ctx, s["tlas"].device_address(), None, None, 0, 0xFF, 0,
                                                        s["rays"].data_ptr(), s["count"], s["hits"].data_ptr(),
                                                        stream))
    hits = s["hits"].view(torch.int32).reshape(s["count"], 8)
    return {"tuv": hits[:, :3].view(torch.float32), "ids": hits[:, 3:]}


@functools.lru_cache(maxsize=1)
def _default_scene_files():
    return assets.standin_assets()


def _frame_scene(case, seed):
    w, h, name = case["width"], case["height"], case["scene"]
    if name == "small":
        return scenes.scene_small(w, h, seed)
    if name == "gallery":
        return scenes.scene_gallery(w, h, seed)
    if name == "default":
        return assets.default_scene(_default_scene_files(), w, h, seed)
    return scenes.scene_full(seed % 1000, w, h, seed)


def _prepare_frame(case, seed):
    scene = _frame_scene(case, seed)
    device = host.Device()
    gpu_scene = host.GpuScene(device, scene)
    frame = host.PerFrameResources(device, gpu_scene, scene.width, scene.height)
    frame.write_uniforms(scene.uniforms)
    return {"case": case, "device": device, "scene": scene, "frame": frame}


def _run_frame(s):
    device, frame, scene = s["device"], s["frame"], s["scene"]
    update = frame.tlas.update_tlas if s["case"]["update"] == "refit" else frame.tlas.rebuild_tlas
    update(device, frame.instances_buffer, frame.num_instances, frame.scratch)
    frame.record(scene.max_trace_depth, scene.shadow_ray_count)
    return frame.image


def _objects_scene(triangles, width, height, rng):
    """Turned tori (one a mirror) and bumpy spheres over a ground grid, seen from a random side: the kind of
    scene the benchmark batches and serves, its unique triangles split 1/2, 1/3, 1/6."""
    def dims(n):
        nv = max(3, int(round(math.sqrt(n / 4.0))))
        return max(3, int(round(n / (2.0 * nv)))), nv

    def model(arrays, diffuse, roughness, name):
        positions, normals, uvs, indices = arrays
        return scenes.Model(positions, normals, uvs, [scenes.Geometry(indices, True, diffuse, roughness)], name)

    cells = max(1, int(round(math.sqrt(triangles / 12))))
    gp, _, guv, gi = scenes.quad_grid(cells, cells, 40.0, 40.0, 8.0, 8.0)
    ground = np.stack([gp[:, 0], np.zeros(len(gp), np.float32), gp[:, 1] - 20.0], -1)
    up = np.tile(np.array([[0.0, 1.0, 0.0]], np.float32), (len(gp), 1))
    models = [model(scenes.torus(1.0, 0.35, *dims(triangles / 2)), scenes.TEX_DIFFUSE_A, scenes.TEX_MR_SHINY, "torus"),
              model(scenes.uv_sphere(*dims(triangles / 3), 1.0, 0.05, int(rng.integers(1 << 20))),
                    scenes.TEX_DIFFUSE_B, scenes.TEX_MR_DEFAULT, "sphere"),
              model((ground, up, guv, gi[:, ::-1]), scenes.TEX_DIFFUSE_B, scenes.TEX_MR_DEFAULT, "ground")]
    xf = np.zeros((11, 3, 4))
    xf[0, :, :3], xf[0, 1, 3] = np.eye(3), -1.2
    xf[1:, :, :3] = _rotations(10, rng) * rng.uniform(0.6, 1.6, (10, 1, 1))
    xf[1:, :, 3] = rng.uniform((-6, -0.5, -6), (6, 2.5, 6), (10, 3))
    which = np.array([2] + [0] * 6 + [1] * 4)
    hit_group = np.full(11, abi.HIT_SHADER_TEXTURED)
    hit_group[1] = abi.HIT_SHADER_MIRROR
    textures = {scenes.TEX_DIFFUSE_A: scenes.solid_rgba32f([0.8, 0.55, 0.3, 1.0]),
                scenes.TEX_DIFFUSE_B: scenes.solid_rgba32f([0.45, 0.5, 0.55, 1.0]),
                scenes.TEX_BLUE_NOISE: scenes.rank_noise_rgba8(int(rng.integers(1 << 20))),
                scenes.TEX_GGX_LUT: scenes.solid_rgba32f([1.0, 1.0, 0.0, 1.0]),
                scenes.TEX_MR_DEFAULT: scenes.metallic_roughness(0.0, 0.6),
                scenes.TEX_MR_SHINY: scenes.metallic_roughness(0.5, 0.3)}
    view = scenes.random_view_uniforms(scenes.Pcg32(int(rng.integers(1 << 30))), width, height)
    return scenes.Scene(models, textures, scenes.instance_records(xf, which, which, hit_group), view, width, height,
                        max_trace_depth=2, shadow_ray_count=2, name="objects")


def _scene_sizes(case):
    """Unique triangles of each scene, from a thirtieth of the case's size up to it."""
    n = case["scenes"]
    return [int(case["triangles"] * 30.0 ** (k / max(1, n - 1) - 1.0)) for k in range(n)]


def _batch_resolutions(n):
    return [RESOLUTIONS[(k * 5 + 2) % len(RESOLUTIONS)] for k in range(n)]


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    device = host.Device()
    if case["packets"]:  # what rt_ctx_autotune picks on the benchmark's batch
        config = abi.RtTraversalConfig(256, 0, 20, abi.RT_TRAVERSAL_PACKET_PRIMARY)
        device.check(device.lib.rt_ctx_set_traversal_config(device.ctx, ctypes.byref(config)))
    flags = abi.RT_BUILD_PREFER_FAST_TRACE | (abi.RT_BUILD_QUANTIZED_NODES if case["nodes"] == "quantised" else 0)
    frames, batch = [], []
    for triangles, (w, h) in zip(_scene_sizes(case), _batch_resolutions(case["scenes"])):
        scene = _objects_scene(triangles, w, h, rng)
        gpu_scene = host.GpuScene(device, scene, blas_flags=flags, own_textures=True)
        frame = host.PerFrameResources(device, gpu_scene, w, h)
        frame.write_uniforms(scene.uniforms)
        frames.append(frame)
        batch.append(host.batch_scene(frame, scene.max_trace_depth, scene.shadow_ray_count))
    return {"case": case, "device": device, "frames": frames, "batch": batch}


def _run_batch(s):
    host.trace_batch(s["device"], s["batch"])
    return [f.image for f in s["frames"]]


def _requests(case):
    """(scene, width, height, shadow rays) of each request, in the order they are sent."""
    return [(k % case["scenes"], *RESOLUTIONS[1:][(k * 3 + 1) % 5], 1 + (k * 5) % 8) for k in range(case["requests"])]


def _prepare_serve(case, seed):
    rng = np.random.default_rng(seed)
    device = host.Device(threadsafe=True)
    gpu_scenes = [host.GpuScene(device, _objects_scene(n, 256, 256, rng), own_textures=True)
                  for n in _scene_sizes(case)]
    server = host.Server(device, 64 << 30, max_batch_requests=32, max_batch_pixels=4 << 20, max_in_flight=2,
                         max_batch_shadow_rays=32 << 20)
    ids = [server.add_scene(g) for g in gpu_scenes]
    requests = []
    for which, w, h, shadows in _requests(case):
        view = scenes.random_view_uniforms(scenes.Pcg32(int(rng.integers(1 << 30))), w, h)
        image = torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True)
        requests.append((ids[which], view, w, h, shadows, image))
    return {"case": case, "device": device, "scenes": gpu_scenes, "server": server, "requests": requests}


def _run_serve(s):
    server = s["server"]
    tickets = [server.submit(i, view, w, h, 2, shadows, image_host=image.data_ptr())
               for i, view, w, h, shadows, image in s["requests"]]
    for t in tickets:
        server.wait(t)
    return [r[-1] for r in s["requests"]]


_PREPARE = {"query": _prepare_query, "frame": _prepare_frame, "batch": _prepare_batch, "serve": _prepare_serve}
_RUN = {"query": _run_query, "frame": _run_frame, "batch": _run_batch, "serve": _run_serve}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# What a pass cannot do without, and what it should give
# ---------------------------------------------------------------------------
RAY_BYTES, HIT_BYTES, INSTANCE_BYTES = 32, 32, 64
TRIANGLE_BYTES = 12 + 6     # its indices, and half a vertex position (a closed mesh has half as many vertices)
BOX_BYTES = {"fp32": 24 + 4, "quantised": 6 + 4}  # a child box and its reference
BOX_FLOPS, TRIANGLE_FLOPS, BUILD_FLOPS = 12, 60, 100


def _trace_work(rays, triangles, instances, nodes="fp32"):
    """Rays that each open one node of eight children per level of the hierarchy and test two triangles;
    no more of the structure is read than it has."""
    levels = math.ceil(math.log(max(8, triangles * instances), 8))
    whole = triangles * (36 + BOX_BYTES[nodes]) + instances * INSTANCE_BYTES
    touched = rays * (levels * 8 * BOX_BYTES[nodes] + 2 * 36)
    return min(whole, touched), rays * (levels * 8 * BOX_FLOPS + 2 * TRIANGLE_FLOPS)


def work(case):
    kind = case["kind"]
    if kind == "query":
        nu, nv = _sphere_grid(case["triangles"])
        t = 2 * nu * nv
        read, flops = _trace_work(case["rays"], t, case["instances"], case["nodes"])
        read += case["rays"] * (RAY_BYTES + HIT_BYTES)
        if case["rebuild"] == "blas":
            read += t * (TRIANGLE_BYTES + 36 + BOX_BYTES[case["nodes"]])  # the mesh in, triangles and boxes out
            flops += t * BUILD_FLOPS
        if case["rebuild"] != "none":
            read += case["instances"] * (INSTANCE_BYTES + 128)
            flops += case["instances"] * BUILD_FLOPS
        return {"bytes": read, "flops": flops}
    if kind == "frame":
        instances, triangles, shadows = {"small": (17, 4098, 1), "gallery": (34, 1100, 2), "default": (105, 47_756, 2),
                                         "full": (256, 20_880, 4)}[case["scene"]]
        frames = [(case["width"], case["height"], shadows, instances, triangles)]
    elif kind == "batch":
        frames = [(w, h, 2, 11, n) for n, (w, h) in zip(_scene_sizes(case), _batch_resolutions(case["scenes"]))]
    else:
        sizes = _scene_sizes(case)
        frames = [(w, h, shadows, 11, sizes[which]) for which, w, h, shadows in _requests(case)]
    total = {"bytes": 0, "flops": 0}
    for w, h, shadows, instances, triangles in frames:
        read, flops = _trace_work(w * h * (1 + shadows), triangles, instances, case.get("nodes", "fp32"))
        total["bytes"] += read + w * h * 4 + instances * INSTANCE_BYTES
        total["flops"] += flops
    return total


def exact(case, seed):
    """The closest hit of every ray in 64 bits, by trying every triangle (t, and the barycentric weights of the
    second and third vertex).  Images are whole numbers, and the larger queries would take minutes: None."""
    if case["kind"] != "query":
        return None
    nu, nv = _sphere_grid(case["triangles"])
    if 2.0 * nu * nv * case["instances"] * case["rays"] > BRUTE_FORCE_PAIRS:
        return None
    positions, indices, transforms, rays = _query_inputs(case, seed)
    v = positions.double()[indices.long()]
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    ray_o = torch.from_numpy(rays["origin"].astype(np.float64)).cuda()
    ray_d = torch.from_numpy(rays["direction"].astype(np.float64)).cuda()
    n = len(rays)
    best = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    best[:, 0] = math.inf
    for m in transforms.astype(np.float64):
        inverse = torch.from_numpy(np.linalg.inv(m[:, :3])).cuda()
        o = (ray_o - torch.from_numpy(m[:, 3]).cuda()) @ inverse.T
        d = ray_d @ inverse.T
        step = max(1, (1 << 25) // len(a))
        for i in range(0, n, step):
            oi, di = o[i:i + step, None, :], d[i:i + step, None, :]
            p = torch.linalg.cross(di, e2[None])
            scale = 1.0 / (p * e1).sum(-1)
            s = oi - a
            u = (s * p).sum(-1) * scale
            q = torch.linalg.cross(s, e1[None].expand_as(s))
            w = (di * q).sum(-1) * scale
            t = (e2 * q).sum(-1) * scale
            t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0), t, torch.full_like(t, math.inf))
            near, k = t.min(1)
            found = torch.stack([near, u.gather(1, k[:, None])[:, 0], w.gather(1, k[:, None])[:, 0]], -1)
            better = near < best[i:i + step, 0]
            best[i:i + step] = torch.where(better[:, None], found, best[i:i + step])
    return {"tuv": best, "ids": None}
