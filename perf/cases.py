"""The work a program does with this library, as cases whose time can be measured.

Each case is one pass of a program through the package's public calls (`bvhtracer_gb300`): tracing
rays against a model from host arrays or from device memory, primaries with one diffuse bounce, an
uneven batch of models, an animated instanced frame, a scene whose objects moved, a rendered image,
a step of the differentiable render (forward, adjoint), an animated model refitted and traced, and a
model loaded.  Geometry and rays come from the package's seeded workloads, at the sizes of its
benchmark and tests and at odd sizes around them.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the pass
    run(state)          one pass, returning its outputs
    work(case)          bytes and operations no implementation can do without
    exact(case, seed)   the outputs in 64 bits, by brute force in torch, where that is quick enough
"""
import ctypes
import functools
import math

import numpy as np
import torch

import bvhtracer_gb300 as bt
from bvhtracer_gb300 import scenes
from bvhtracer_gb300.frames import AnimatedScene


def listed():
    return [
        # An editor's pick or one 8x8 tile of the renderer: 64 rays from a host array, the smallest call.
        {"name": "pick_tile", "kind": "host", "mesh": "soup", "size": 4096, "rays": "camera", "count": 64},
        # The 640 x 640 frame of the 4,096-triangle soup, rays and hits in device memory.
        {"name": "soup_frame", "kind": "device", "mesh": "soup", "size": 4096, "rays": "camera", "count": 409600},
        # The renderer's own use: an image of a scene of shaded instances (path tracer, normal shading), to host memory.
        {"name": "render_scene", "kind": "render", "instances": 24, "size": 5, "width": 640, "height": 480},
        # A full-HD frame of the 81,920-triangle model with one diffuse bounce per hit.
        {"name": "bounce_1080p", "kind": "bounce", "size": 6, "width": 1920, "height": 1080, "host": False},
        # The same from ordinary host arrays at a small odd size, as a caller without a GPU pipeline has it.
        {"name": "bounce_host", "kind": "bounce", "size": 5, "width": 641, "height": 479, "host": True},
        # A serving batch: many models of very different sizes, many ray counts, one call.
        {"name": "uneven_batch", "kind": "batch", "models": 16, "max_tris": 200000, "max_rays": 262144},
        # One frame of the animated scene at 720p: wobble, refit, instance motion, TLAS rebuild, trace + bounce.
        {"name": "instanced_720p", "kind": "frame", "instances": 256, "levels": "4,5,6", "width": 1280, "height": 720},
        # A scene of many small objects moved by the host, rebuilt and traced from host arrays.
        {"name": "moved_scene", "kind": "scene", "instances": 1000, "size": 3, "width": 321, "height": 241},
        # The gradient of a 512 x 512 Lambertian render of a 327,680-triangle mesh: update, forward, adjoint.
        {"name": "lambert_512", "kind": "lambert", "size": 7, "width": 512, "height": 512, "loss": False},
        # The same on a small mesh at an odd size, with the loss read back, as a training loop does.
        {"name": "lambert_small", "kind": "lambert", "size": 5, "width": 129, "height": 97, "loss": True},
        # An animated model: new vertices in device memory, refit, a small frame.
        {"name": "refit_trace", "kind": "refit", "size": 5, "width": 320, "height": 200},
        # A model loaded: the BVH built, uploaded, and a first thumbnail traced.
        {"name": "load_model", "kind": "load", "mesh": "sphere", "size": 6, "count": 3072},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "bounce", "batch", "frame", "scene", "render", "lambert", "refit", "load"])
    if kind in ("host", "device", "load"):
        mesh = rng.choice(["soup", "sphere"])
        size = _log(rng, 300, 20000) if mesh == "soup" else rng.randint(2, 6)
        if kind == "load":
            return {"kind": kind, "mesh": mesh, "size": size, "count": _log(rng, 1, 4096)}
        most = 20000 if kind == "host" else 400000
        return {"kind": kind, "mesh": mesh, "size": size, "rays": rng.choice(["camera", "random"]),
                "count": _log(rng, 1 if kind == "host" else 1000, most)}
    if kind == "bounce":
        host = rng.random() < 0.4
        return {"kind": kind, "size": rng.randint(3, 6), "width": _log(rng, 40, 800 if host else 1920),
                "height": _log(rng, 40, 600 if host else 1080), "host": host}
    if kind == "batch":
        return {"kind": kind, "models": rng.randint(2, 16), "max_tris": _log(rng, 4000, 200000),
                "max_rays": _log(rng, 16384, 262144)}
    if kind == "frame":
        lo = rng.randint(2, 4)
        return {"kind": kind, "instances": rng.randint(16, 256), "levels": "%d,%d,%d" % (lo, lo + 1, lo + 2),
                "width": _log(rng, 100, 1280), "height": _log(rng, 60, 720)}
    if kind == "scene":
        return {"kind": kind, "instances": _log(rng, 3, 1000), "size": rng.randint(1, 4),
                "width": _log(rng, 16, 400), "height": _log(rng, 16, 300)}
    if kind == "render":
        return {"kind": kind, "instances": _log(rng, 1, 64), "size": rng.randint(1, 5),
                "width": _log(rng, 32, 640), "height": _log(rng, 32, 480)}
    if kind == "lambert":
        return {"kind": kind, "size": rng.randint(3, 6), "width": _log(rng, 32, 512), "height": _log(rng, 32, 512),
                "loss": rng.random() < 0.5}
    return {"kind": kind, "size": rng.randint(3, 6), "width": _log(rng, 32, 640), "height": _log(rng, 32, 400)}


# ---- inputs -------------------------------------------------------------------------------------

_icosphere = functools.lru_cache(maxsize=None)(scenes.icosphere)


def _sphere(level, seed):
    dirs, faces = _icosphere(level)
    return scenes.Mesh(dirs, scenes.displaced_radius(dirs, seed), faces)


def _triangles(case, seed):
    if case["mesh"] == "soup":
        return scenes.soup(case["size"], seed, scale=_scale(case))
    return _sphere(case["size"], seed).triangles()


def _scale(case):
    """Larger soups keep the density of the 4,096-triangle one."""
    return (case["size"] / 4096.0) ** (1.0 / 3.0) if case["mesh"] == "soup" else 1.0


def _rays(case, seed):
    n, s = case["count"], _scale(case)
    if case.get("rays") == "random":
        return scenes.sphere_rays(n, seed, box=10.0 * s if case["mesh"] == "soup" else 4.0)
    side = int(math.ceil(math.sqrt(n) / 8.0) * 8)
    if case["mesh"] == "soup":
        return scenes.plane_rays(side, side, (0.0, 0.0, -18.0 * s), -15.0 * s, s, s)[:n]
    return scenes.look_at_rays(side, side, (0.0, 0.0, -3.0), (0.0, 0.0, 0.0), 45.0)[:n]


def _camera_eye(seed, dist):
    """A viewpoint somewhere around the model, off its planes of symmetry."""
    a, e = scenes.uniform(seed, 90, 2)
    a, e = 2.0 * math.pi * a, 0.1 + 0.4 * e
    return (dist * math.cos(e) * math.sin(a), dist * math.sin(e), -dist * math.cos(e) * math.cos(a))


def _camera_rays(case, seed, dist=3.0, fov=45.0):
    return scenes.look_at_rays(case["width"], case["height"], _camera_eye(seed, dist), (0.0, 0.0, 0.0), fov)


def _attitude(case, seed):
    """Position, forward, right and up of a camera that sees the scene's box from outside."""
    eye = np.array(_camera_eye(seed, 60.0 * (case["instances"] / 256.0) ** (1.0 / 3.0)))
    fwd = -eye / np.linalg.norm(eye)
    right = np.cross(fwd, (0.0, 1.0, 0.0))
    right /= np.linalg.norm(right)
    return tuple(eye), tuple(fwd), tuple(right), tuple(np.cross(right, fwd))


def _transforms(n, seed):
    """Random rigid motions with a uniform scale in a box that keeps 256 objects' density."""
    cfg = scenes.instanced_animation(seed, n, 8, 8, levels=(1,))["instances"]
    rot = cfg["rot0"].astype(np.float64)
    s = cfg["scale"].astype(np.float64)[:, None, None]
    t = cfg["trans"].astype(np.float64) * (n / 256.0) ** (1.0 / 3.0)
    m = np.zeros((n, 4, 4))
    m[:, :3, :3] = rot * s
    m[:, :3, 3] = t
    m[:, 3, 3] = 1.0
    inv = np.linalg.inv(m)
    return (np.ascontiguousarray(m.transpose(0, 2, 1), np.float32).reshape(n, 16),
            np.ascontiguousarray(inv.transpose(0, 2, 1), np.float32).reshape(n, 16))


def _batch_shape(case):
    """Triangle and ray counts, log-uniform; the seed makes the models and rays, not their number."""
    nt, nr = scenes.batch_specs(0, case["models"], (1000, case["max_tris"]), (4096, case["max_rays"]))
    # the largest model and the largest ray set are always there, in different scenes
    nt[0], nr[-1] = case["max_tris"], case["max_rays"]
    return nt, nr


# ---- device memory: torch tensors handed over by their address ------------------------------------

class _Dev:
    def __init__(self, tensor):
        self.tensor = tensor

    @property
    def ptr(self):
        return ctypes.c_void_p(self.tensor.data_ptr())


def _to_device(a):
    return _Dev(torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda())


def _hit_buffer(n):
    return _Dev(torch.zeros((n, 5), dtype=torch.int32, device="cuda"))


def _device_hits(buf):
    f = buf.tensor.view(torch.float32)
    return {"t": f[:, 0], "uv": f[:, 1:3], "id": buf.tensor[:, 3:]}


def _host_hits(h):
    return {"t": h["t"], "u": h["u"], "v": h["v"], "prim": h["prim"].view(np.int32), "inst": h["inst"].view(np.int32)}


# ---- a program's state -----------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    return bt.Context(0)


class _State:
    """What the program keeps between passes; its models are given back with it."""

    def __init__(self, case):
        self.case = case
        self.ctx = _context()
        self.models, self.scenes, self.meshes, self.graphs = [], [], [], []

    def model(self, tris):
        bvh = self.ctx.build_bvh(tris)
        blas = self.ctx.upload_blas(bvh, tris)
        self.models.append(blas)
        return blas

    def diff_mesh(self, verts, faces, normals):
        mesh = bt.DiffMesh(self.ctx, verts, faces, normals)
        self.meshes.append(mesh)
        self.models.append(mesh.blas)
        return mesh

    def __del__(self):
        try:
            self.ctx.sync()
            for g in self.graphs:
                self.ctx.graph_free(g)
            for m in self.meshes:
                self.ctx.lib.bvhgpu_mesh_free(self.ctx.h, m.id)
            for x in self.scenes + self.models:
                x.free()
        except Exception:
            pass


def prepare(case, seed):
    s = _State(case)
    ctx, kind = s.ctx, case["kind"]
    if kind in ("host", "device"):
        s.blas = s.model(_triangles(case, seed))
        s.rays = _rays(case, seed + 1)
        s.n = len(s.rays)
        if kind == "device":
            s.d_rays, s.d_hits = _to_device(s.rays), _hit_buffer(s.n)
    elif kind == "bounce":
        s.blas = s.model(_sphere(case["size"], seed).triangles())
        s.rays = _camera_rays(case, seed)
        s.n, s.seed = len(s.rays), seed & 0x7FFFFFFF
        if not case["host"]:
            s.d_rays, s.d_h0, s.d_h1 = _to_device(s.rays), _hit_buffer(s.n), _hit_buffer(s.n)
    elif kind == "batch":
        nt, nr = _batch_shape(case)
        items, rays, at = np.zeros(len(nt), bt.BATCH_ITEM), [], 0
        for i in range(len(nt)):
            tris, r = _batch_model(i, int(nt[i]), int(nr[i]), seed)
            items[i]["blas"], items[i]["ray_offset"], items[i]["ray_count"] = s.model(tris).id, at, len(r)
            rays.append(r)
            at += len(r)
        s.items, s.n = items, at
        s.d_rays, s.d_hits = _to_device(np.concatenate(rays)), _hit_buffer(at)
    elif kind == "frame":
        levels = tuple(int(x) for x in case["levels"].split(","))
        cfg = scenes.instanced_animation(seed, case["instances"], case["width"], case["height"], levels)
        s.anim = AnimatedScene(ctx, cfg, bounce_seed=seed & 0x7FFFFFFF)
        s.meshes += s.anim.meshes
        s.models += [m.blas for m in s.anim.meshes]
        s.scenes.append(s.anim.scene)
        s.anim.d_hits0, s.anim.d_hits1 = _hit_buffer(s.anim.n), _hit_buffer(s.anim.n)
        s.anim.frame_async()
        ctx.sync()
        s.anim.set_time(0.0)
        s.graphs.append(s.anim.capture())
    elif kind == "scene":
        blas = s.model(_sphere(case["size"], seed).triangles())
        s.scene = ctx.scene([blas] * case["instances"])
        s.scenes.append(s.scene)
        s.xf, s.inv = _transforms(case["instances"], seed)
        s.rays = _camera_rays(case, seed, dist=60.0 * (case["instances"] / 256.0) ** (1.0 / 3.0), fov=60.0)
    elif kind == "render":
        mesh = _sphere(case["size"], seed)
        tris = mesh.triangles()
        bvh, perm = ctx.build_bvh(tris, perm=True)
        blas = ctx.upload_blas(bvh, tris)
        s.models.append(blas)
        blas.set_shading(normals=mesh.dirs[mesh.faces].astype(np.float32).reshape(-1, 9)[perm])
        xf, inv = _transforms(case["instances"], seed)
        s.scene = ctx.scene([blas] * case["instances"], xf, inv)
        s.scenes.append(s.scene)
        s.camera = bt.Camera.symmetric_fov(60.0, case["width"] / case["height"], 0.1, 100.0, *_attitude(case, seed))
    elif kind == "lambert":
        verts, faces, normals, _, rays, light = _lambert(case, seed)
        s.mesh = s.diff_mesh(verts, faces, normals)
        s.light, s.n = light, len(rays)
        s.d_rays, s.d_hits = _to_device(rays), _hit_buffer(s.n)
        s.d_image = _Dev(torch.zeros(s.n, device="cuda"))
        s.d_target = _Dev(torch.from_numpy(_target(s.n, seed)).cuda())
        s.d_grad = _Dev(torch.zeros((len(verts), 3), device="cuda"))
    elif kind == "refit":
        tris = _sphere(case["size"], seed).triangles()
        s.blas = s.model(tris)
        s.d_tris = _to_device(_moved(tris, seed))
        rays = _camera_rays(case, seed)
        s.n = len(rays)
        s.d_rays, s.d_hits = _to_device(rays), _hit_buffer(s.n)
    elif kind == "load":
        s.tris = _triangles(case, seed)
        s.rays = _rays(case, seed + 1)
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx, kind = s.case, s.ctx, s.case["kind"]
    if kind == "host":
        return _host_hits(s.blas.intersect(s.rays))
    if kind == "device":
        s.blas.intersect_async(s.d_rays, s.n, s.d_hits)
        return _device_hits(s.d_hits)
    if kind == "bounce":
        if case["host"]:
            h0, h1, n = s.blas.trace_bounce(s.rays, s.seed, bt.MODE_PERSISTENT)
            return [_host_hits(h0), _host_hits(h1), n]
        s.blas.trace_bounce_async(s.d_rays, s.n, s.seed, bt.MODE_PERSISTENT, s.d_h0, s.d_h1)
        return [_device_hits(s.d_h0), _device_hits(s.d_h1)]
    if kind == "batch":
        ctx.trace_batch_async(s.items, s.d_rays, s.n, bt.MODE_PERSISTENT, s.d_hits)
        return _device_hits(s.d_hits)
    if kind == "frame":
        s.anim.launch()
        return [_device_hits(s.anim.d_hits0), _device_hits(s.anim.d_hits1)]
    if kind == "scene":
        s.scene.set_transforms(s.xf, s.inv)
        s.scene.rebuild()
        return _host_hits(s.scene.intersect(s.rays))
    if kind == "render":
        rgba, rays = s.scene.render(s.camera, case["width"], case["height"], bt.ACC_NORMAL, bt.SHADER_RADIANCE,
                                    lookup=bt.LOOKUP_HIT_OBJECT)
        return [rgba, rays]
    if kind == "lambert":
        # the adjoint adds into the gradient: cleared on the library's own stream
        ctx.check(ctx.lib.bvhgpu_memset_device(ctx.h, s.d_grad.ptr, 0, 4 * s.d_grad.tensor.numel(), None))
        s.mesh.update_async()
        s.mesh.forward_async(s.d_rays, s.n, s.light, s.d_image, s.d_hits)
        s.mesh.adjoint_async(s.d_rays, s.n, s.light, s.d_hits, s.d_image, s.d_target, s.d_grad)
        out = {"image": s.d_image.tensor, "hits": _device_hits(s.d_hits), "grad": s.d_grad.tensor}
        if case["loss"]:
            out["loss"] = bt.mse_loss(ctx, s.d_image, s.d_target, s.n)
        return out
    if kind == "refit":
        s.blas.update_vertices_async(s.d_tris)
        s.blas.refit_async()
        s.blas.intersect_async(s.d_rays, s.n, s.d_hits)
        return _device_hits(s.d_hits)
    tris = s.tris.copy()  # the build reorders the triangles in place
    bvh, perm = ctx.build_bvh(tris, perm=True)
    blas = ctx.upload_blas(bvh, tris)
    hits = blas.intersect(s.rays)
    blas.free()
    nodes = bvh.nodes  # zero past the nodes used
    return {"box": np.concatenate([nodes["bounds_min"], nodes["bounds_max"]], axis=1),
            "child": np.stack([nodes["left_first"], nodes["primitive_count"]], axis=1).view(np.int32),
            "perm": perm.view(np.int32), "used": bvh.nodes_used, "hits": _host_hits(hits)}


def _batch_model(i, ntris, nrays, seed):
    """scenes.batch_scene's model and rays, with this file's cached spheres."""
    sseed = (seed * 1000 + i) & 0x7FFFFFFF
    if i % 2 == 0:
        case = {"mesh": "soup", "size": ntris}
        prim = {"rays": "camera", "count": nrays // 2, **case}
    else:
        case = {"mesh": "sphere", "size": int(np.clip(np.round(math.log(ntris / 20.0, 4)), 1, 8))}
        prim = {"rays": "camera", "count": nrays // 2, **case}
    box = 10.0 * _scale(case)
    return _triangles(case, sseed), np.concatenate([_rays(prim, sseed), scenes.sphere_rays(nrays - nrays // 2, sseed + 7, box=box)])


def _lambert(case, seed):
    """scenes.lambert_scene at any size, with this file's cached spheres (all lengths times 10)."""
    mesh = _sphere(case["size"], seed)
    verts = (mesh.dirs * (10.0 * mesh.radius)[:, None]).astype(np.float32)
    rays = _camera_rays(case, seed, dist=30.0)
    eye = np.array(_camera_eye(seed, 30.0))  # the light stands beside the camera and above it
    right = np.cross((0.0, 1.0, 0.0), -eye / 30.0)
    light = (eye + 20.0 * right / np.linalg.norm(right) + (0.0, 20.0, 0.0)).astype(np.float32)
    return verts, mesh.faces.astype(np.uint32), mesh.dirs.astype(np.float32), None, rays, light


def _target(n, seed):
    return (0.5 + 0.25 * scenes.uniform(seed, 91, n)).astype(np.float32)


def _moved(tris, seed):
    """The next pose of the model: every corner moved along its radius by the same smooth wave."""
    v = tris.reshape(-1, 3).astype(np.float64)
    w = scenes.normal(seed, 92, 3)
    v = v * (1.0 + 0.05 * np.sin(3.0 * (v @ w)))[:, None]
    return np.ascontiguousarray(v.astype(np.float32).reshape(-1, 9))


# ---- work -----------------------------------------------------------------------------------------

def _tris(case):
    return case["size"] if case.get("mesh") == "soup" else 20 * 4 ** case["size"]


def _trace_flops(rays, tris):
    """A walk down a balanced binary tree (two boxes a level) and one triangle, per ray."""
    return rays * (40.0 * math.log2(max(2, tris)) + 60.0)


def work(case):
    kind = case["kind"]
    if kind in ("host", "device", "load"):
        n, t = case["count"], _tris(case)
        more = 4.0 * t + 36.0 * t if kind == "load" else 0.0
        return {"bytes": 52.0 * n + 36.0 * t + more, "flops": _trace_flops(n, t)}
    if kind == "batch":
        nt, nr = _batch_shape(case)
        return {"bytes": float(52 * nr.sum() + 36 * nt.sum()),
                "flops": float(sum(_trace_flops(int(r), int(t)) for r, t in zip(nr, nt)))}
    n = case["width"] * case["height"]
    if kind == "frame":
        t = sum(20 * 4 ** int(x) for x in case["levels"].split(","))
        return {"bytes": 72.0 * n + 36.0 * t + 128.0 * case["instances"], "flops": _trace_flops(1.3 * n, 3 * t)}
    if kind == "scene":
        return {"bytes": 52.0 * n + 36.0 * _tris(case) + 128.0 * case["instances"],
                "flops": _trace_flops(n, _tris(case) * case["instances"])}
    t = _tris(case)
    if kind == "render":  # no rays in: the image out, the model and its normals in
        return {"bytes": 4.0 * n + 72.0 * t + 128.0 * case["instances"], "flops": _trace_flops(n, t * case["instances"])}
    if kind == "bounce":
        return {"bytes": 72.0 * n + 36.0 * t, "flops": _trace_flops(1.3 * n, t)}
    if kind == "refit":
        return {"bytes": 52.0 * n + 36.0 * t, "flops": _trace_flops(n, t)}
    # render: rays in, hits and image out, target in; mesh: faces, vertices and normals in, gradient out
    return {"bytes": 60.0 * n + 12.0 * t + 18.0 * t, "flops": _trace_flops(n, t) + 200.0 * n}


# ---- the same in 64 bits ----------------------------------------------------------------------------

_FLT_MAX = float(np.finfo(np.float32).max)


def _closest64(tris, rays):
    """(t, u, v, triangle) of every ray's closest hit by brute force in 64 bits; a miss has t = FLT_MAX,
    u = v = 0, triangle -1.  A triangle counts where |det| >= 1e-4, 0 <= u <= 1, 0 <= v, u + v <= 1
    and 1e-4 < t < the ray's own limit."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = torch.from_numpy(tris.astype(np.float64)).to(dev).view(-1, 3, 3)
    v0, e1, e2 = T[:, 0], T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]
    c12 = torch.linalg.cross(e1, e2)  # det = -d . c12, t = s . c12 / det
    o_all = torch.from_numpy(rays["origin"].astype(np.float64)).to(dev)
    d_all = torch.from_numpy(rays["direction"].astype(np.float64)).to(dev)
    n, m = len(rays), len(T)
    best = [torch.full((n,), _FLT_MAX, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev),
            torch.zeros(n, dtype=torch.float64, device=dev), torch.full((n,), -1, dtype=torch.int64, device=dev)]
    step = max(1, (1 << 26) // m)
    for a in range(0, n, step):
        o, d = o_all[a:a + step], d_all[a:a + step]
        # every triple product as matrix products over the rays: s = o - v0
        det = -(d @ c12.T)
        sn = o @ c12.T - (v0 * c12).sum(1)
        od = torch.linalg.cross(o, d)
        # u det = s . (d x e2) = e2 . (s x d) = e2 . (o x d) - e2 . (v0 x d) = e2 . (o x d) - d . (e2 x v0)
        ud = od @ e2.T - d @ torch.linalg.cross(e2, v0).T
        # v det = d . (s x e1) = -e1 . (s x d)
        vd = -(od @ e1.T - d @ torch.linalg.cross(e1, v0).T)
        t, u, v = sn / det, ud / det, vd / det
        ok = (det.abs() >= 1e-4) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-4)
        t = torch.where(ok, t, torch.full_like(t, _FLT_MAX))
        tm, k = t.min(dim=1)
        hit = tm < _FLT_MAX
        at = torch.arange(len(k), device=dev)
        best[0][a:a + step] = tm
        best[1][a:a + step] = torch.where(hit, u[at, k], 0.0)
        best[2][a:a + step] = torch.where(hit, v[at, k], 0.0)
        best[3][a:a + step] = torch.where(hit, k, -1)
    return best


def _hits64(tris, rays, host):
    t, u, v, _ = _closest64(tris, rays)
    if host:
        return {"t": t, "u": u, "v": v, "prim": None, "inst": None}
    return {"t": t, "uv": torch.stack([u, v], dim=1), "id": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host", "device"):
        if case["count"] * _tris(case) > 2e10:
            return None
        return _hits64(_triangles(case, seed), _rays(case, seed + 1), kind == "host")
    if kind == "load":
        if case["count"] * _tris(case) > 2e10:
            return None
        return {"box": None, "child": None, "perm": None, "used": None, "hits": _hits64(_triangles(case, seed), _rays(case, seed + 1), True)}
    if kind in ("batch", "frame", "scene", "render"):
        return None  # too many pairs of a ray and a triangle; an image's bytes have no 64-bit value
    n = case["width"] * case["height"]
    if n * _tris(case) > 2e10:
        return None
    if kind == "bounce":  # the bounce directions follow from the 32-bit primary hits: primaries only
        h = _hits64(_sphere(case["size"], seed).triangles(), _camera_rays(case, seed), case["host"])
        none = {k: None for k in h}
        return [h, none, None] if case["host"] else [h, none]
    if kind == "refit":
        return _hits64(_moved(_sphere(case["size"], seed).triangles(), seed), _camera_rays(case, seed), False)
    return _lambert64(case, seed)


def _lambert64(case, seed):
    """Image, hits and gradient of the Lambertian render in 64 bits: the hit's triangle by brute force,
    its t, u, v and the shading differentiated by autograd with the visible triangle held fixed."""
    verts, faces, normals, _, rays, light = _lambert(case, seed)
    tris = verts[faces].reshape(-1, 9)
    t0, u0, v0, k = _closest64(tris, rays)
    dev = t0.device
    hit = k >= 0
    f = torch.from_numpy(faces.astype(np.int64)).to(dev)[k[hit]]
    V = torch.from_numpy(verts.astype(np.float64)).to(dev).requires_grad_(True)
    N = torch.from_numpy(normals.astype(np.float64)).to(dev)
    o = torch.from_numpy(rays["origin"].astype(np.float64)).to(dev)[hit]
    d = torch.from_numpy(rays["direction"].astype(np.float64)).to(dev)[hit]
    L = torch.from_numpy(light.astype(np.float64)).to(dev)
    a, b, c = V[f[:, 0]], V[f[:, 1]], V[f[:, 2]]
    e1, e2, s = b - a, c - a, o - a
    p = torch.linalg.cross(d, e2)
    det = (e1 * p).sum(1)
    q = torch.linalg.cross(s, e1)
    u, v, t = (s * p).sum(1) / det, (d * q).sum(1) / det, (e2 * q).sum(1) / det
    n = N[f[:, 0]] * (1 - u - v)[:, None] + N[f[:, 1]] * u[:, None] + N[f[:, 2]] * v[:, None]
    ln = L - (o + d * t[:, None])
    I = torch.clamp((n * ln).sum(1) / (n.norm(dim=1) * ln.norm(dim=1)), min=0.0)
    image = torch.zeros(len(rays), dtype=torch.float64, device=dev).masked_scatter(hit, I)
    target = torch.from_numpy(_target(len(rays), seed).astype(np.float64)).to(dev)
    loss = ((image - target) ** 2).mean()
    loss.backward()
    out = {"image": image.detach(), "hits": {"t": t0, "uv": torch.stack([u0, v0], dim=1), "id": None}, "grad": V.grad}
    if case["loss"]:
        out["loss"] = float(loss.detach())
    return out
