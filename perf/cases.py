"""Performance cases: the work a renderer gives this library, through its
Python entry points (Context, Scene, Batch), from one picking query to a full
1080p frame. Each case is one dict; `prepare` makes what a program holds
before the call, `run` is the call (or the two or three calls) of one frame.

Geometry is the seeded synthetic scenes of foundation_gb300.scenes (the
sphere scene, the Cornell box, the triangle soups, the terrain), kept per
process; everything that changes from frame to frame (rays, cameras, vertex
positions, textures, network inputs) comes from the seed.
"""
import functools
import math

import numpy as np
import torch

import foundation_gb300 as fg
from foundation_gb300 import rt, scenes

TREE_SPLIT = dict(spatial_splits=True, split_budget=8.0, sah_collapse=True)  # static scenes: the best tree
TREE_GPU = dict(gpu_build=True, cluster=True, sah_collapse=True)            # dynamic scenes: built on the GPU
CACHE = dict(train_paths=65536, train_steps=6, batch=16384, learning_rate=1e-2, weight_average=0.98,
             specular_alpha=0.05)
CACHE_WARMUP = 16  # training-only frames before the first cache frame


def listed():
    return [
        # a few host rays against a small scene: mouse picking, a probe; latency is all of it
        dict(name="pick_host", kind="trace", scene="spheres", query="closest", mem="host", rays=1000),
        # the visibility buffer of a 1024 x 1024 camera and one shadow ray per pixel
        dict(name="frame_1024", kind="frame", scene="spheres", width=1024, height=1024),
        # the bounce rays of a path tracer: incoherent closest hits on 256k triangles
        dict(name="incoherent_cornell", kind="trace", scene="cornell", query="closest", mem="device", rays=8388608),
        # incoherent closest hits on a million overlapping triangles (the tree does not fit L2)
        dict(name="incoherent_soup", kind="trace", scene="soup", query="closest", mem="device", rays=4194304),
        # a terrain with a thousand instanced spheres, two-level traversal
        dict(name="instanced", kind="instanced", grid=512, instances=1024, rays=2097152),
        # many small scenes, closest-hit and any-hit batches, one graph launch
        dict(name="batch_48", kind="batch", scenes=48, max_tris=65536, max_rays=131072),
        # a host application's whole call on pinned buffers, copies included
        dict(name="host_pinned", kind="trace", scene="cornell", query="closest", mem="pinned", rays=4194304),
        # a progressive 1080p frame of the plain path tracer
        dict(name="render_1080p", kind="render", width=1920, height=1080, spp=2, cache=False),
        # a 1080p frame that ends its paths in the radiance cache, and trains it
        dict(name="cache_frame_1080p", kind="render", width=1920, height=1080, spp=1, cache=True),
        # the cache network by itself: forward, loss and backward of one training batch
        dict(name="cache_gradient", kind="gradient", samples=16384),
        # moving geometry: a million triangles uploaded, built on the GPU, traced and dropped
        dict(name="rebuild_1m", kind="rebuild", grid=725, rays=524288),
        # the raster pass of the reference renderer at 1080p
        dict(name="raster_1080p", kind="raster", width=1920, height=1080, tex=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "frame", "instanced", "batch", "render", "render", "gradient",
                       "rebuild", "raster"])
    if kind == "trace":
        mem = rng.choice(["device", "device", "host", "pinned"])
        top = {"device": 8388608, "host": 65536, "pinned": 4194304}[mem]
        return dict(kind=kind, scene=rng.choice(["spheres", "cornell", "soup"]), query=rng.choice(["closest", "any"]),
                    mem=mem, rays=_log(rng, 100, top))
    if kind == "frame":
        return dict(kind=kind, scene=rng.choice(["spheres", "cornell"]), width=_log(rng, 64, 1600),
                    height=_log(rng, 64, 1200))
    if kind == "instanced":
        return dict(kind=kind, grid=rng.randint(65, 512), instances=_log(rng, 16, 1024), rays=_log(rng, 1000, 2097152))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 48), max_tris=_log(rng, 2000, 65536),
                    max_rays=_log(rng, 8000, 131072))
    if kind == "render":
        if rng.random() < 0.3:
            return dict(kind=kind, width=rng.randint(1000, 1920), height=rng.randint(600, 1080), spp=1, cache=True)
        return dict(kind=kind, width=_log(rng, 96, 1920), height=_log(rng, 54, 1080), spp=rng.randint(1, 2), cache=False)
    if kind == "gradient":
        return dict(kind=kind, samples=_log(rng, 257, 65536))
    if kind == "rebuild":
        return dict(kind=kind, grid=_log(rng, 33, 725), rays=_log(rng, 1000, 524288))
    return dict(kind=kind, width=_log(rng, 64, 1920), height=_log(rng, 36, 1080), tex=rng.randint(16, 512))


# ---- geometry (seeded, the same for every state) ----------------------------
@functools.lru_cache(maxsize=None)
def _scene(name):
    if name == "spheres":
        return scenes.icosphere_scene()
    if name == "cornell":
        return scenes.cornell_scene()
    return scenes.soup_scene(1 << 20)


@functools.lru_cache(maxsize=8)
def _terrain(grid, instances=0):
    return scenes.terrain_scene(grid=grid, instances=max(instances, 1))


@functools.lru_cache(maxsize=4)
def _batch_scenes(count, max_tris):
    nt = scenes.log_uniform_ints(count, 1000, max_tris, 2, 1 << 50)
    base = np.concatenate([[0], np.cumsum(nt[:-1])])
    return [scenes.soup_scene(int(n), seed=2, stream_base=int(b)) for n, b in zip(nt, base)]


def _upload(ctx, name):
    sc = _scene(name)
    # the soup's spatial-split tree takes the host seconds: the GPU build stands in for it
    opts = {"spheres": {}, "cornell": TREE_SPLIT, "soup": TREE_GPU}[name]
    return ctx.upload(sc.verts, sc.idx, **opts)


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rays(n, lo, hi, seed, any_hit=False):
    """Incoherent rays: origins uniform in the box, directions uniform on the
    sphere; any-hit queries are segments between two points of the box."""
    g = _gen(seed)
    lo = torch.tensor(lo, dtype=torch.float32, device="cuda")
    ext = torch.tensor(hi, dtype=torch.float32, device="cuda") - lo
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = lo + torch.rand((n, 3), generator=g, device="cuda") * ext
    r[:, 3] = 0.0
    if any_hit:
        r[:, 4:7] = lo + torch.rand((n, 3), generator=g, device="cuda") * ext - r[:, 0:3]
        r[:, 7] = 1.0
    else:
        d = torch.randn((n, 3), generator=g, device="cuda")
        r[:, 4:7] = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)
        r[:, 7] = math.inf
    return r


def _jitter(seed, k, scale):
    return float(np.random.default_rng([seed, k]).uniform(-scale, scale))


def _camera(base, seed):
    eye = [e + _jitter(seed, k, 0.02) for k, e in enumerate(base["eye"])]
    return dict(base, eye=tuple(eye))


class _Pinned:
    """Page-locked bytes as an array whose views keep the memory."""

    def __init__(self, nbytes):
        self.buf = rt.PinnedBuffer(nbytes)
        self.__array_interface__ = dict(self.buf.view(np.uint8, (nbytes,)).__array_interface__)


def _pinned(nbytes):
    return np.asarray(_Pinned(nbytes))


class State:
    """One context and what the case holds on it; closes the context when it goes."""

    def __init__(self):
        self.ctx = fg.Context(0)

    def __del__(self):
        try:
            torch.cuda.synchronize()
            if getattr(self, "batch", None) is not None:
                self.batch.close()
            self.ctx.close()
        except Exception:
            pass


def prepare(case, seed):
    s = State()
    ctx, kind = s.ctx, case["kind"]
    s.case = case
    if kind == "trace":
        sc = _scene(case["scene"])
        s.any = case["query"] == "any"
        s.scene = _upload(ctx, case["scene"])
        rays = _rays(case["rays"], *sc.bounds, seed, s.any)
        n = case["rays"]
        if case["mem"] == "device":
            s.rays = rays
            s.out = torch.empty(n if s.any else 2 * n, dtype=torch.uint8 if s.any else torch.int32, device="cuda")
        elif case["mem"] == "host":
            s.rays, s.out = rays.cpu().numpy(), None
        else:
            s.rays = _pinned(32 * n).view(np.float32).reshape(n, 8)
            s.rays[:] = rays.cpu().numpy()
            s.out = _pinned(n if s.any else 8 * n).view(np.uint8 if s.any else rt.HIT_DTYPE)
    elif kind == "frame":
        sc = _scene(case["scene"])
        s.scene = _upload(ctx, case["scene"])
        base = scenes.CORNELL_CAMERA if case["scene"] == "cornell" else dict(eye=(0.0, 0.0, 5.0), target=(0.0, 0.0, 0.0))
        n = case["width"] * case["height"]
        cam = _camera(base, seed)
        s.rays = torch.from_numpy(scenes.camera_rays(case["width"], case["height"], cam["eye"], cam["target"])).cuda()
        s.out = torch.empty(2 * n, dtype=torch.int32, device="cuda")
        # one segment per pixel from a point of the scene to a light above it
        s.shadow = _rays(n, *sc.bounds, seed, True)
        light = torch.tensor(sc.bounds[1], dtype=torch.float32, device="cuda")
        s.shadow[:, 4:7] = light * torch.tensor([0.2, 0.99, 0.2], device="cuda") - s.shadow[:, 0:3]
        s.occluded = torch.empty(n, dtype=torch.uint8, device="cuda")
    elif kind == "instanced":
        grid, count = case["grid"], case["instances"]
        tr = _terrain(grid)
        nt = 2 * (grid - 1) ** 2
        s.ground = ctx.upload(tr.verts[:grid * grid], tr.idx[:nt], gpu_build=True, sah_collapse=True)
        sv, sf = scenes.icosphere(4)
        s.sphere = ctx.upload(sv.astype(np.float32), sf, margin_scale=128)
        rng = np.random.default_rng(4)
        x, z, rad = rng.uniform(0, 1, count), rng.uniform(0, 1, count), rng.uniform(0.002, 0.02, count)
        y = scenes.value_noise(x, z, 3) + 0.5 * rad
        inst = [(s.ground, np.eye(3, 4, dtype=np.float32), 0)]
        for k in range(count):
            m = np.concatenate([np.eye(3) * rad[k], [[x[k]], [y[k]], [z[k]]]], 1).astype(np.float32)
            inst.append((s.sphere, m, nt + k * len(sf)))
        s.scene = ctx.instances(inst)
        s.rays = _rays(case["rays"], *tr.bounds, seed)
        s.out = torch.empty(2 * case["rays"], dtype=torch.int32, device="cuda")
    elif kind == "batch":
        nr = scenes.log_uniform_ints(case["scenes"], 4096, case["max_rays"], 2, (1 << 50) + 4096)
        jobs, total, at = [], int(nr.sum()), 0
        s.hits = torch.zeros(2 * total, dtype=torch.int32, device="cuda")
        s.occluded = torch.zeros(total, dtype=torch.uint8, device="cuda")
        for k, sc in enumerate(_batch_scenes(case["scenes"], case["max_tris"])):
            scene, n = ctx.upload(sc.verts, sc.idx, sah_collapse=True), int(nr[k])
            closest = _rays(n, *sc.bounds, seed + 1009 * k)
            half = torch.from_numpy(scenes.cube_camera_rays(n // 2)).cuda()
            closest[:n // 2] = half  # half coherent camera rays, half random ones
            for q, rays in ((rt.QUERY_CLOSEST, closest), (rt.QUERY_ANY, _rays(n, *sc.bounds, seed + 1009 * k + 1, True))):
                jobs.append((scene, rays, s.occluded[at:at + n] if q else s.hits[2 * at:2 * (at + n)], q))
            at += n
        torch.cuda.synchronize()
        s.batch = fg.Batch(ctx, jobs)
    elif kind == "render":
        sc = _scene("cornell")
        s.scene = _upload(ctx, "cornell")
        s.scene.set_materials(sc.tri_material, scenes.material_records(sc))
        s.scene.set_lights(scenes.light_records(sc))
        s.cam = _camera(scenes.CORNELL_CAMERA, seed)
        s.seed = seed
        s.out = torch.empty(case["width"] * case["height"] * 3, dtype=torch.float32, device="cuda")
        if case["cache"]:
            ctx.cache_create(s.scene, seed=seed, **CACHE)
            for f in range(CACHE_WARMUP):
                ctx.render(s.scene, case["width"], case["height"], 1, s.cam, seed=seed + 100 + f, cache=True,
                           train_only=True)
            ctx.sync()
    elif kind == "gradient":
        rng = np.random.default_rng(seed)
        sv, sf = scenes.icosphere(2)
        s.scene = ctx.upload(sv.astype(np.float32), sf)
        ctx.cache_create(s.scene, seed=seed)
        ctx.cache_set_weights(_weights(seed))
        s.features, s.targets = _samples(case["samples"], seed)
    elif kind == "rebuild":
        tr = _terrain(case["grid"])
        s.verts = _moved(tr.verts, seed)
        s.idx = tr.idx
        s.rays = _rays(case["rays"], *tr.bounds, seed)
        s.out = torch.empty(2 * case["rays"], dtype=torch.int32, device="cuda")
    else:
        rng = np.random.default_rng(seed)
        t = 0.3 + 3.0 * rng.random()
        s.uniforms = rt.raster_uniforms(t, case["width"] / case["height"])
        s.texture = rng.integers(0, 256, (case["tex"], case["tex"], 4), dtype=np.uint8)
        s.out = torch.empty(case["width"] * case["height"] * 4, dtype=torch.uint8, device="cuda")
    return s


def _moved(verts, seed):
    """The mesh a frame later: a wave through its heights."""
    ph = np.random.default_rng(seed).uniform(0, 6.28)
    v = verts.copy()
    v[:, 1] += (0.01 * np.sin(9.0 * v[:, 0] + ph)).astype(np.float32)
    return v


_SHAPES = [(96, 64), (64, 64), (64, 64), (64, 64), (64, 64), (64, 3)]  # the cache network, input to output


def _weights(seed):
    rng = np.random.default_rng([seed, 7])
    return np.concatenate([rng.uniform(-1, 1, k * n) * math.sqrt(6.0 / k) for k, n in _SHAPES]).astype(np.float32)


def _samples(n, seed):
    """Encoded cache points (sine / cosine bands, directions, materials) and radiance targets."""
    rng = np.random.default_rng([seed, 8])
    x = np.sin(rng.uniform(-math.pi, math.pi, (n, 96)))
    x[:, 72:] = rng.uniform(-1.0, 1.0, (n, 24))
    x[:, 82:] = 0.0
    return x.astype(np.float32), rng.exponential(0.5, (n, 3)).astype(np.float32)


def _hits(out):
    v = out.view(-1, 2)
    return {"prim": v[:, 0], "t": v[:, 1].view(torch.float32)}


def run(s):
    case, ctx = s.case, s.ctx
    kind = case["kind"]
    if kind == "trace":
        call = s.scene.any if s.any else s.scene.closest
        out = call(s.rays, s.out)
        if case["mem"] == "device":
            return {"occluded": out} if s.any else _hits(out)
        return {"occluded": out} if s.any else {"prim": out["prim"].view(np.int32), "t": out["t"]}
    if kind == "frame":
        s.scene.closest(s.rays, s.out)
        s.scene.any(s.shadow, s.occluded)
        return {**_hits(s.out), "occluded": s.occluded}
    if kind == "instanced":
        return _hits(s.scene.closest(s.rays, s.out))
    if kind == "batch":
        s.batch.launch()
        return {**_hits(s.hits), "occluded": s.occluded}
    if kind == "render":
        return ctx.render(s.scene, case["width"], case["height"], case["spp"], s.cam, seed=s.seed, out=s.out,
                          cache=case["cache"])
    if kind == "gradient":
        grad, loss = ctx.cache_gradient(s.features, s.targets)
        return {"grad": grad, "loss": loss}
    if kind == "rebuild":
        scene = ctx.upload(s.verts, s.idx, **TREE_GPU)
        hits = _hits(scene.closest(s.rays, s.out))
        scene.close()
        return hits
    return ctx.raster_draw(case["width"], case["height"], *s.uniforms, s.texture, out=s.out)


def _log8(n):
    return max(1.0, math.log(max(n, 2)) / math.log(8))


def _trace_work(tris, rays, out_bytes):
    """Rays in, results out, the triangles (vertices and id) once; per ray one
    path of 8 box tests per level of an 8-wide tree and one triangle test."""
    return {"bytes": rays * (32 + out_bytes) + 40 * min(tris, 4 * rays), "flops": rays * (_log8(tris) * 8 * 12 + 50)}


def work(case):
    kind = case["kind"]
    tris = {"spheres": 82944, "cornell": 256012, "soup": 1 << 20}
    if kind == "trace":
        return _trace_work(tris[case["scene"]], case["rays"], 1 if case["query"] == "any" else 8)
    if kind == "frame":
        a, b = (_trace_work(tris[case["scene"]], case["width"] * case["height"], o) for o in (8, 1))
        return {"bytes": a["bytes"] + b["bytes"], "flops": a["flops"] + b["flops"]}
    if kind == "instanced":
        return _trace_work(2 * (case["grid"] - 1) ** 2 + 5120, case["rays"], 8)
    if kind == "batch":
        nr = scenes.log_uniform_ints(case["scenes"], 4096, case["max_rays"], 2, (1 << 50) + 4096)
        nt = scenes.log_uniform_ints(case["scenes"], 1000, case["max_tris"], 2, 1 << 50)
        all_ = [_trace_work(int(t), int(n), o) for t, n in zip(nt, nr) for o in (8, 1)]
        return {k: float(sum(w[k] for w in all_)) for k in ("bytes", "flops")}
    if kind == "render":
        # about 7 rays a path (3.3 closest, 3.3 shadow); with the cache 2 + 2 and one network evaluation;
        # the scene once and the image once
        pix = case["width"] * case["height"]
        rays = pix * case["spp"] * (4 if case["cache"] else 7)
        flops = rays * (_log8(256012) * 8 * 12 + 50)
        if case["cache"]:
            flops += pix * 45440 + 6 * 16384 * 3 * 45440 + 65536 * 7 * (_log8(256012) * 8 * 12 + 50)
        return {"bytes": 40 * 256012 + 12 * pix, "flops": flops}
    if kind == "gradient":
        n = case["samples"]
        return {"bytes": n * (96 + 3) * 4 + 2 * 22720 * 4, "flops": n * 3 * 2 * 22720}
    if kind == "rebuild":
        g = case["grid"]
        nt = 2 * (g - 1) ** 2 + 5120
        w = _trace_work(nt, case["rays"], 8)
        # vertices and indices in; boxes, codes and one sort pass, triangles and about a fifth of a node each out
        return {"bytes": w["bytes"] + 12 * g * g + 12 * nt + nt * (32 + 24 + 48 + 16), "flops": w["flops"] + nt * 500}
    pix = case["width"] * case["height"]
    return {"bytes": 4 * pix + 4 * case["tex"] ** 2, "flops": pix * 100}


def _brute_t(v, idx, rays):
    """Nearest t of every ray over all triangles, in 64 bits (Moeller-Trumbore)."""
    p = torch.from_numpy(v[idx.astype(np.int64)]).cuda().double()
    a, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    best = []
    for r in torch.as_tensor(rays).cuda().double().split(128):
        o, d = r[:, None, 0:3], r[:, None, 4:7].expand(-1, len(a), -1)
        q = torch.linalg.cross(d, e2[None].expand_as(d))
        det = (q * e1).sum(-1)
        s = o - a
        u = (s * q).sum(-1) / det
        w = torch.linalg.cross(s, e1[None].expand_as(s))
        b = (d * w).sum(-1) / det
        t = (e2 * w).sum(-1) / det
        ok = (det != 0) & (u >= 0) & (b >= 0) & (u + b <= 1) & (t >= r[:, None, 3]) & (t <= r[:, None, 7])
        best.append(torch.where(ok, t, math.inf).amin(1))
    return torch.cat(best)


def exact(case, seed):
    if case["kind"] == "trace" and case["query"] == "closest":
        sc = _scene(case["scene"])
        if case["rays"] * len(sc.idx) > 1 << 29:
            return None
        return {"prim": None, "t": _brute_t(sc.verts, sc.idx, _rays(case["rays"], *sc.bounds, seed))}
    if case["kind"] == "gradient":
        x, y = (torch.from_numpy(a).cuda().double() for a in _samples(case["samples"], seed))
        w, params, at = torch.from_numpy(_weights(seed)).cuda().double(), [], 0
        for k, n in _SHAPES:
            params.append(w[at:at + k * n].view(k, n).clone().requires_grad_(True))
            at += k * n
        h = x
        for m in params[:-1]:
            h = (h @ m).relu()
        out = h @ params[-1]
        loss = ((out - y) ** 2 / (out.detach() ** 2 + 0.01)).mean()
        loss.backward()
        return {"grad": torch.cat([m.grad.reshape(-1) for m in params]), "loss": loss.detach()}
    return None
