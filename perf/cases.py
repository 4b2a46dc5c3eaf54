"""Timed cases of the ray-query backend: scene builds and nearest-hit queries through the
public entry points (portablert_gb300.backend, .batch and .serve), over the range of sizes
that programs use them with.

A case is a dict of plain values.  ``prepare`` makes what a program has in hand before the
call (triangles and rays on the GPU, or in host memory where the call takes host arrays; the
backend with its scene; a batch or a server), ``run`` makes one pass through the framework
and returns every record it wrote, field by field.

Kinds of case:

* ``host``   ``B200Backend.nearest_hits`` on numpy rays: the call portableRT's own interface
             makes, records in a new host array.
* ``query``  ``nearest_hits_dev``: rays and records stay on the GPU (a path tracer's bounce).
* ``build``  ``set_tris_dev`` (``set_tris`` when the triangles are on the host) and the
             first rays on the new scene: geometry that changes from frame to frame.
* ``camera`` ``nearest_hits_camera`` and ``shade_lambert``: one frame of the examples.
* ``batch``  ``Batch.run_graph``: many scenes built and queried as one CUDA graph.
* ``serve``  ``Server``: requests of mixed sizes against resident scenes.

Scenes: ``soup`` (triangles about random centres: no coherence), ``field`` (a heightfield,
two triangles per quad), ``clusters`` (Gaussian clusters of small triangles) and ``ball`` (a
closed bumpy mesh, the examples' bunny in size).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from portablert_gb300 import _lib, backend, hitreg
from portablert_gb300.batch import Batch, make_query
from portablert_gb300.serve import Server

ALL = "uv,t,primitive_id,p,valid"
NO_P = "uv,t,primitive_id,valid"
HIT = "t,primitive_id,valid"

_stream_of_program = None


def _stream():
    """The stream a program queues its device work on (one for the process)."""
    global _stream_of_program
    if _stream_of_program is None:
        _stream_of_program = torch.cuda.Stream()
    return _stream_of_program


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # A few picks or shadow tests against a small object, from host arrays: latency.
        {"name": "host_picks", "kind": "host", "scene": "soup", "tris": 512, "rays": 1000,
         "ray_kind": "aimed", "tags": HIT},
        # The small configuration: 4,096 triangles, 65,536 rays.
        {"name": "query_small", "kind": "query", "scene": "soup", "tris": 4096, "rays": 65536,
         "ray_kind": "aimed", "tags": ALL, "compressed": False, "leaf_size": 1},
        # The main configuration: a 1,048,576-triangle heightfield, a 1920 x 1080 pinhole
        # camera's rays and cosine-distributed secondary rays from what they hit.
        {"name": "query_field", "kind": "query", "scene": "field", "tris": 1048576,
         "rays": 6267904, "ray_kind": "path", "tags": ALL, "compressed": False,
         "leaf_size": 1},
        # The precision configuration's scene (larger than L2) with a quarter of its rays.
        {"name": "query_clusters", "kind": "query", "scene": "clusters", "tris": 8388608,
         "rays": 4194304, "ray_kind": "random", "tags": NO_P, "compressed": False,
         "leaf_size": 1},
        # The memory-saving options in use: 8-bit nodes, leaves of several triangles; odd
        # sizes.
        {"name": "query_compressed", "kind": "query", "scene": "clusters", "tris": 1000003,
         "rays": 1000003, "ray_kind": "random", "tags": NO_P, "compressed": True,
         "leaf_size": 4},
        # portableRT's std::vector call at a camera's size, rays and records in host memory.
        {"name": "host_field", "kind": "host", "scene": "field", "tris": 1048576,
         "rays": 2073600, "ray_kind": "camera", "tags": ALL},
        # A small object rebuilt each frame.
        {"name": "build_small", "kind": "build", "scene": "soup", "tris": 4096, "rays": 4096,
         "ray_kind": "aimed", "tags": ALL, "host_tris": False},
        # A mid-sized animated mesh, triangles from host memory, odd sizes.
        {"name": "build_mid", "kind": "build", "scene": "field", "tris": 65790, "rays": 76799,
         "ray_kind": "camera", "tags": HIT, "host_tris": True},
        # The main configuration's scene build.
        {"name": "build_large", "kind": "build", "scene": "field", "tris": 1048576,
         "rays": 65536, "ray_kind": "camera", "tags": ALL, "host_tris": False},
        # The bunny example: 4,968 triangles, a 2048 x 2048 sensor, Lambert shading.
        {"name": "camera_frame", "kind": "camera", "scene": "ball", "tris": 4968,
         "width": 2048, "height": 2048, "tags": HIT},
        # The batch configuration, an eighth of its scenes: sizes log-uniform in 16..65,536
        # triangles and 64..262,144 rays.
        {"name": "batch_graph", "kind": "batch", "scenes": 512, "max_tris": 65536,
         "max_rays": 262144, "mix": 3, "tags": NO_P},
        # The serving configuration in waves: requests of 1,024..262,144 rays on 16 scenes.
        {"name": "serve_mixed", "kind": "serve", "scenes": 16, "max_tris": 262144,
         "requests": 48, "max_rays": 262144, "mix": 9, "tags": NO_P},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random):
    kind = rng.choice(("host", "query", "query", "build", "build", "camera", "batch", "serve"))
    tags = rng.choice((ALL, NO_P, HIT))
    scene, ray_kind = rng.choice((("soup", "aimed"), ("field", "camera"), ("field", "path"),
                                  ("clusters", "random")))
    # Rays in a dense soup cross boxes all the way through it, so it stays small; few rays
    # meet a sparse cluster, so there are many of both.
    low, top = (64, 16384) if scene == "soup" else (64, 2097152)
    few = 64
    if scene == "clusters":
        low, few = 131072, 16384
    if kind == "host":
        return {"kind": kind, "scene": scene, "tris": _log_int(rng, low, top),
                "rays": _log_int(rng, few, 1048576), "ray_kind": ray_kind, "tags": tags}
    if kind == "query":
        compressed = rng.random() < 0.25
        return {"kind": kind, "scene": scene, "tris": _log_int(rng, low, top),
                "rays": _log_int(rng, max(few, 256), 2097152), "ray_kind": ray_kind,
                "tags": tags, "compressed": compressed,
                "leaf_size": rng.choice((1, 2, 4, 8)) if compressed else rng.choice((1, 1, 4))}
    if kind == "build":
        tris = _log_int(rng, low, top)
        return {"kind": kind, "scene": scene, "tris": tris,
                "rays": _log_int(rng, max(few, tris // 16, 256), 131072),
                "ray_kind": ray_kind, "tags": tags, "host_tris": rng.random() < 0.5}
    if kind == "camera":
        w = _log_int(rng, 160, 2048)
        return {"kind": kind, "scene": "ball", "tris": _log_int(rng, 256, 65536), "width": w,
                "height": max(1, int(w * rng.uniform(0.5, 1.0))), "tags": HIT}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 4, 256),
                "max_tris": _log_int(rng, 256, 32768), "max_rays": _log_int(rng, 256, 131072),
                "mix": rng.randrange(1000), "tags": NO_P}
    return {"kind": kind, "scenes": _log_int(rng, 2, 12), "max_tris": _log_int(rng, 512, 65536),
            "requests": _log_int(rng, 2, 32), "max_rays": _log_int(rng, 2048, 131072),
            "mix": rng.randrange(1000), "tags": rng.choice((ALL, NO_P))}


# ---------------------------------------------------------------- scenes and rays


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + stream)


def _uniform(g, a, b, *shape):
    return a + (b - a) * torch.rand(shape, generator=g, device="cuda")


def _unit(g, n):
    v = torch.randn((n, 3), generator=g, device="cuda")
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-20)


def _soup(seed, n):
    """Centres in [-1, 1]^3, vertices within 0.05 of them."""
    g = _generator(seed, 1)
    c = _uniform(g, -1.0, 1.0, n, 1, 3)
    return (c + _uniform(g, -0.05, 0.05, n, 3, 3)).reshape(n, 9)


def _field(seed, n):
    """Sum of eight sinusoids over [-4, 4] x [-2, 2], about twice as many quads in x as in
    z; the last row is cut so that there are n triangles."""
    nz = max(1, math.isqrt(n // 4))
    nx = max(1, -(-n // (2 * nz)))
    r = random.Random(int(seed))
    x = torch.linspace(-4.0, 4.0, nx + 1, device="cuda", dtype=torch.float64)
    z = torch.linspace(-2.0, 2.0, nz + 1, device="cuda", dtype=torch.float64)
    h = torch.zeros((nz + 1, nx + 1), device="cuda", dtype=torch.float64)
    for _ in range(8):
        f, phase, a = 0.5 + 7.5 * r.random(), 2 * math.pi * r.random(), 2 * math.pi * r.random()
        h += torch.sin(f * (x[None, :] * math.cos(a) + z[:, None] * math.sin(a)) + phase) / f
    v = torch.stack([x[None, :].expand_as(h), h, z[:, None].expand_as(h)], -1).float()
    v00, v10, v01, v11 = v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]
    t = torch.stack([torch.cat([v00, v10, v01], -1), torch.cat([v10, v11, v01], -1)], 2)
    return t.reshape(-1, 9)[:n].contiguous()


def _clusters(seed, n):
    """256 Gaussian clusters in [-10, 10]^3, edges within 0.02."""
    g = _generator(seed, 2)
    centre = _uniform(g, -10.0, 10.0, 256, 3)
    sigma = _uniform(g, 0.1, 1.0, 256, 1)
    c = torch.randint(0, 256, (n,), generator=g, device="cuda")
    v0 = centre[c] + sigma[c] * torch.randn((n, 3), generator=g, device="cuda")
    e = _uniform(g, -0.02, 0.02, n, 2, 3)
    return torch.cat([v0, v0 + e[:, 0], v0 + e[:, 1]], 1).contiguous()


def _ball(seed, n):
    """A closed bumpy sphere of radius about 0.06 (the bunny's size) in latitude rings."""
    nv = max(2, math.isqrt(n // 4))
    nu = max(3, -(-n // (2 * nv)))
    r = random.Random(int(seed))
    a = torch.linspace(0.0, math.pi, nv + 1, device="cuda", dtype=torch.float64)[:, None]
    b = torch.linspace(0.0, 2 * math.pi, nu + 1, device="cuda", dtype=torch.float64)[None, :]
    rad = torch.full((nv + 1, nu + 1), 0.06, device="cuda", dtype=torch.float64)
    for _ in range(6):
        ka, kb = r.randrange(1, 7), r.randrange(0, 7)
        rad += 0.006 * r.random() * torch.sin(ka * a) * torch.cos(kb * b + 6.28 * r.random())
    v = torch.stack([rad * torch.sin(a) * torch.cos(b), rad * torch.cos(a).expand_as(rad),
                     rad * torch.sin(a) * torch.sin(b)], -1).float()
    v00, v10, v01, v11 = v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]
    t = torch.stack([torch.cat([v00, v10, v01], -1), torch.cat([v10, v11, v01], -1)], 2)
    return t.reshape(-1, 9)[:n].contiguous()


_SCENES = {"soup": _soup, "field": _field, "clusters": _clusters, "ball": _ball}


def _camera_size(n):
    """Width and height (about 16 : 9) of an image of at least n pixels."""
    h = max(1, math.isqrt(n * 9 // 16))
    return -(-n // h), h


def _camera_rays(n):
    """Pinhole rays from (0, 3, -6) towards the origin, 60 degrees, row by row."""
    w, h = _camera_size(n)
    eye = torch.tensor([0.0, 3.0, -6.0], device="cuda", dtype=torch.float64)
    fwd = -eye / eye.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device="cuda",
                                                 dtype=torch.float64))
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    th = math.tan(math.radians(30.0))
    px = (2.0 * (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w - 1.0) * th * w / h
    py = (1.0 - 2.0 * (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h) * th
    d = fwd + px[None, :, None] * right + py[:, None, None] * up
    d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)[:n].float()
    return torch.cat([eye.float().expand_as(d), d], 1).contiguous()


def _path_rays(b, tris, seed, n):
    """The first third camera rays, the rest cosine-distributed about the normals of what
    those hit, from 0.01 off the surface."""
    first = _camera_rays(max(1, n // 3))
    lay = hitreg.layout(("primitive_id", "p", "valid"))
    rec = torch.zeros((len(first), lay.size), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    b.nearest_hits_dev(first.data_ptr(), len(first), rec.data_ptr(), lay.tags)
    b.sync()
    f = _fields(rec, lay)
    hit = torch.nonzero(f["valid"].reshape(-1)).reshape(-1)
    if len(hit) == 0:
        return _camera_rays(n)
    m = n - len(first)
    src = hit[torch.arange(m, device="cuda") % len(hit)]
    t = tris[f["primitive_id"][src].reshape(-1).long()]
    nrm = torch.linalg.cross(t[:, 3:6] - t[:, 0:3], t[:, 6:9] - t[:, 0:3])
    nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    nrm = torch.where((nrm * first[src, 3:6]).sum(1, keepdim=True) > 0, -nrm, nrm)
    d = nrm + 0.999 * _unit(_generator(seed, 4), m)
    d = d / d.norm(dim=1, keepdim=True)
    second = torch.cat([f["p"][src] + 0.01 * nrm, d], 1)
    return torch.cat([first, second]).contiguous()


def _aimed_rays(seed, n):
    """From the sphere of radius 3 at points of [-0.5, 0.5]^3."""
    g = _generator(seed, 5)
    o = 3.0 * _unit(g, n)
    d = _uniform(g, -0.5, 0.5, n, 3) - o
    return torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).contiguous()


def _random_rays(seed, n):
    """Origins in [-12, 12]^3, directions uniform on the sphere."""
    g = _generator(seed, 6)
    return torch.cat([_uniform(g, -12.0, 12.0, n, 3), _unit(g, n)], 1).contiguous()


def _rays(case, b, tris, seed):
    n, kind = case["rays"], case["ray_kind"]
    if kind == "camera":
        return _camera_rays(n)
    if kind == "path":
        return _path_rays(b, tris, seed, n)
    return _aimed_rays(seed, n) if kind == "aimed" else _random_rays(seed, n)


# ---------------------------------------------------------------- preparation


def _fields(rec, lay):
    """Views of the fields of a record buffer (records x bytes, uint8)."""
    f32, i32 = rec.view(torch.float32), rec.view(torch.int32)
    out = {}
    if "uv" in lay.tags:
        out["uv"] = f32[:, lay.off_u // 4:lay.off_v // 4 + 1]
    if "t" in lay.tags:
        out["t"] = f32[:, lay.off_t // 4]
    if "primitive_id" in lay.tags:
        out["primitive_id"] = i32[:, lay.off_pid // 4]
    if "valid" in lay.tags:
        out["valid"] = rec[:, lay.off_valid]
    if "p" in lay.tags:
        out["p"] = f32[:, lay.off_px // 4:lay.off_px // 4 + 3]
    return out


def _records(case, n):
    lay = hitreg.layout(case["tags"].split(","))
    rec = torch.zeros((n, lay.size), dtype=torch.uint8, device="cuda")
    return rec, lay


def _mix_sizes(case):
    """Per-scene triangle counts and ray counts (or per-request ray counts), log-uniform."""
    r = random.Random(case["mix"])
    tris = [_log_int(r, 16 if case["kind"] == "batch" else 256, case["max_tris"])
            for _ in range(case["scenes"])]
    if case["kind"] == "batch":
        return tris, [_log_int(r, 64, case["max_rays"]) for _ in range(case["scenes"])]
    return tris, [(r.randrange(case["scenes"]), _log_int(r, 1024, case["max_rays"]))
                  for _ in range(case["requests"])]


def _scene_soups(seed, sizes):
    return torch.cat([_soup(1000 * int(seed) + i, n) for i, n in enumerate(sizes)]).contiguous()


def prepare(case, seed):
    b = backend.B200Backend(0)
    b.init()
    s = {"case": case, "b": b}
    kind = case["kind"]
    if kind in ("batch", "serve"):
        _prepare_many(case, seed, s)
        torch.cuda.synchronize()
        return s
    tris = _SCENES[case["scene"]](seed, case["tris"])
    torch.cuda.synchronize()
    b.set_option("leaf_size", case.get("leaf_size", 1))
    b.set_tris_dev(tris.data_ptr(), len(tris))
    if case.get("compressed"):
        b.set_option("node_format", 1)
    s["tags"] = tuple(case["tags"].split(","))
    if kind == "camera":
        _prepare_camera(case, s)
    else:
        rays = _rays(case, b, tris, seed)
        if kind == "host":
            s["rays"] = rays.cpu().numpy()
        else:
            s["rays"] = rays
            s["rec"], lay = _records(case, len(rays))
            s["out"] = _fields(s["rec"], lay)
        if kind == "build":
            s["tris"] = tris.cpu().numpy() if case["host_tris"] else tris
    torch.cuda.synchronize()
    return s


def _prepare_camera(case, s):
    cam = _lib.Camera()
    cam.width, cam.height, cam.form = case["width"], case["height"], _lib.CAMERA_PLANE
    cam.pos[:] = [0.0, -0.02, -0.3]
    cam.sensor_size, cam.sensor_dist = 0.05, 0.05
    cam.sensor_z = float(np.float32(-0.3) + np.float32(0.05))
    n = case["width"] * case["height"]
    s["cam"] = cam
    s["rec"], lay = _records(case, n)
    s["rgba"] = torch.zeros((n, 4), dtype=torch.uint8, device="cuda")
    s["out"] = dict(_fields(s["rec"], lay), rgba=s["rgba"])


def _prepare_many(case, seed, s):
    b = s["b"]
    sizes, work = _mix_sizes(case)
    s["tris"] = _scene_soups(seed, sizes)
    s["off"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    rays_of = [w if case["kind"] == "batch" else w[1] for w in work]
    at = np.concatenate([[0], np.cumsum(rays_of)]).astype(np.int64)
    total = int(at[-1])
    rays = _aimed_rays(seed, total)
    s["rec"], lay = _records(case, total)
    tags = lay.tags
    if case["kind"] == "batch":
        s["rays"] = rays
        s["out"] = _fields(s["rec"], lay)
        s["queries"] = (_lib.Query * len(sizes))(*[
            make_query(i, rays.data_ptr() + 24 * int(at[i]), n,
                       s["rec"].data_ptr() + lay.size * int(at[i]), tags)
            for i, n in enumerate(rays_of)])
        s["batch"] = Batch(b)
        torch.cuda.synchronize()
        # As the autotuner does: the traversal's pool sized for the depth that the build
        # reaches.
        _run_batch(s)
        s["batch"].sync()
        b.set_option("pool_depth", int(s["batch"].stat("depth")))
        return
    torch.cuda.synchronize()
    s["rays"] = rays.cpu().pin_memory()
    s["rec"] = torch.zeros((total, lay.size), dtype=torch.uint8).pin_memory()
    s["out"] = _fields(s["rec"], lay)
    b.set_option("serve_persistent", 0)
    s["server"] = Server(b, s["tris"].data_ptr(), s["off"], 1 << 30, lanes=4)
    s["requests"] = [(scene, s["rays"].data_ptr() + 24 * int(at[i]), n, tags,
                      s["rec"].data_ptr() + lay.size * int(at[i]))
                     for i, (scene, n) in enumerate(work)]


# ---------------------------------------------------------------- one pass


def _run_host(s):
    h = s["b"].nearest_hits(s["rays"], s["tags"])
    return {f: h[f] for f in h.dtype.names}


def _run_query(s):
    r = s["rays"]
    s["b"].nearest_hits_dev(r.data_ptr(), r.shape[0], s["rec"].data_ptr(), s["tags"],
                            _stream().cuda_stream)
    return s["out"]


def _run_build(s):
    t = s["tris"]
    if isinstance(t, np.ndarray):
        s["b"].set_tris(t)
    else:
        s["b"].set_tris_dev(t.data_ptr(), t.shape[0])
    return _run_query(s)


def _run_camera(s):
    st = _stream().cuda_stream
    s["b"].nearest_hits_camera(s["cam"], s["rec"].data_ptr(), s["tags"], st)
    s["b"].shade_lambert(s["rec"].data_ptr(), s["tags"], s["rgba"].data_ptr(), cam=s["cam"],
                         stream=st)
    return s["out"]


def _run_batch(s):
    s["batch"].run_graph(s["tris"].data_ptr(), s["off"], s["queries"], _stream().cuda_stream)
    return s["out"]


def _run_serve(s):
    srv = s["server"]
    for ticket in [srv.submit_ptr(*r) for r in s["requests"]]:
        srv.wait(ticket)
    return s["out"]


_RUN = {"host": _run_host, "query": _run_query, "build": _run_build, "camera": _run_camera,
        "batch": _run_batch, "serve": _run_serve}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------- work and exact values


def work(case):
    """Bytes: rays read (24 B, none for a camera), records and pixels written, and the
    triangles (36 B; at most one per ray where the scene is not built in the pass) read,
    built scenes' triangle records (48 B) and nodes (256 B for each 7 triangles) written.
    Operations: per ray one path from the root to a triangle (eight box tests of 21 on each
    of log8 n levels, one triangle test of 45); per triangle built its bounds and one
    comparison for each of log2 n levels (30 + log2 n)."""
    kind = case["kind"]
    rec = hitreg.layout(case["tags"].split(",")).size
    if kind in ("batch", "serve"):
        sizes, w = _mix_sizes(case)
        pairs = ([(n, m) for n, m in zip(sizes, w)] if kind == "batch"
                 else [(sizes[i], m) for i, m in w])
    elif kind == "camera":
        pairs = [(case["tris"], case["width"] * case["height"])]
    else:
        pairs = [(case["tris"], case["rays"])]
    built = kind in ("build", "batch")
    total = {"bytes": 0.0, "flops": 0.0}
    for n, m in pairs:
        levels = max(1, math.ceil(math.log(max(n, 2), 8)))
        total["bytes"] += m * (rec + (4 if kind == "camera" else 24))
        total["bytes"] += n * (36 + 48 + 256 / 7) if built else 36 * min(n, m)
        total["flops"] += m * (levels * 8 * 21 + 45)
        total["flops"] += n * (30 + math.log2(max(n, 2))) if built else 0
    return total


def exact(case, seed):
    """Every ray against every triangle in 64 bits: the smallest t of the triangles that the
    Moller-Trumbore test accepts and whose bounding box the ray passes.  None where that
    takes too long."""
    if case["kind"] not in ("host", "query", "build") or case["tris"] * case["rays"] > 3e8:
        return None
    if case["ray_kind"] == "path":
        return None  # these rays come from a query
    tris = _SCENES[case["scene"]](seed, case["tris"])
    rays = _rays(case, None, tris, seed)
    v = tris.double().reshape(-1, 3, 3)
    lo, hi = v.amin(1), v.amax(1)
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    step = max(1, 8_000_000 // len(v))
    parts = []
    for r in rays.double().split(step):
        o, d = r[:, None, :3], r[:, None, 3:]
        t1, t2 = (lo - o) / d, (hi - o) / d
        near, far = torch.minimum(t1, t2).amax(-1), torch.maximum(t1, t2).amin(-1)
        h = torch.linalg.cross(d.expand(-1, len(v), -1), e2.expand(len(r), -1, -1))
        det = (e1 * h).sum(-1)
        s = o - v0
        q = torch.linalg.cross(s, e1.expand(len(r), -1, -1))
        u, w = (s * h).sum(-1) / det, (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (far >= 0) & (near <= far) & (det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1)
        t, k = torch.where(ok, t, math.inf).min(1)
        miss = torch.isinf(t)
        uw = torch.stack([u.gather(1, k[:, None])[:, 0], w.gather(1, k[:, None])[:, 0]], 1)
        uw[miss] = 0.0
        parts.append((uw, t, r[:, :3] + t[:, None] * r[:, 3:]))
    uw, t, p = (torch.cat(x) for x in zip(*parts))
    tags = case["tags"].split(",")
    if case["kind"] == "host":
        cols = {"u": uw[:, 0], "v": uw[:, 1], "t": t, "px": p[:, 0], "py": p[:, 1], "pz": p[:, 2]}
        names = hitreg.layout(tags).numpy_dtype().names
        return {f: cols.get(f) for f in names}
    cols = {"uv": uw, "t": t, "p": p}
    return {f: cols.get(f) for f in tags}
