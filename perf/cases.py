"""The work a program has this library do, as measurable cases.

Each case is one call, or one short sequence of calls, of the public Python
host (lambda_b200.renderer.Context over include/lambda_gpu.h):

  render    a frame of one scene, into host memory (Context.render) or device
            memory (Context.render_device)
  batch     many small jobs, or the tiles of one frame, in one launch
            (Context.render_batch_device)
  adjoint   image-loss gradients by path replay (Context.adjoint_device)
  inverse   one iteration of an inverse-rendering loop on host arrays:
            Context.update_materials, render, adjoint
  rays      closest-hit and shadow-ray queries (Context.trace, trace_any)
  upload    a new scene and its first preview frame (Context.upload, render)
  tonemap   the filmic tone map of a frame in device memory
            (lgpu_tonemap_noalloc) or host memory (Context.tonemap)

Scenes are seeded synthetic ones of the kinds of lambda_b200.synth: the box
room, the scene with every object, material and light kind, instances of a
displaced icosphere on a ground quad, the box room filled with such
instances, and the thin-film / albedo inverse-rendering scene.  The seed sets
materials, spectra, placements and the random streams; the meshes of one
subdivision are shared by a process, as a loader shares them.
"""
import functools
import math
import tempfile

import numpy as np
import torch

from lambda_b200 import _lib as L
from lambda_b200 import synth
from lambda_b200.renderer import Context
from lambda_b200.scene import (Camera, FlatScene, LightDef, Material, Object, SceneData, SpectralConfig, Transform,
                               TriMeshData, blinn_init, load_nls)


# ---- the cases -------------------------------------------------------------------

def listed():
    return [
        # the smallest call: a thumbnail at the renderer's default settings (4 spp, 4 bounces, p = 0.5)
        dict(name="thumbnail", op="render", scene="box", w=64, h=64, spp=4, bounces=4, p=0.5, k=16, host=True,
             film64=False),
        # the box-room configuration: an ordinary small render through the host call
        dict(name="box_room", op="render", scene="box", w=256, h=256, spp=16, bounces=8, p=0.8, k=4, host=True,
             film64=False),
        # a reference-quality still: thin lens, every object, material and light kind, FP64 film
        dict(name="mixed_fp64", op="render", scene="mixed", w=361, h=289, spp=48, bounces=12, p=0.8, k=8, host=True,
             film64=True),
        # the benchmark frame: 21 M instanced triangles, full HD
        dict(name="frame_hd", op="render", scene="instanced", inst=64, sub=7, w=1920, h=1080, spp=64, bounces=32,
             p=0.8, k=16, host=False, film64=False),
        # an interactive frame of odd size with few samples
        dict(name="frame_ragged", op="render", scene="instanced", inst=9, sub=5, w=1021, h=577, spp=6, bounces=16,
             p=0.8, k=8, host=False, film64=False),
        # small jobs of many scenes in one launch (dataset generation)
        dict(name="batch_jobs", op="batch", kind="jobs", jobs=14, sub=5, size=192, spp=12, bounces=16, p=0.8, k=4),
        # one larger frame as tile jobs
        dict(name="batch_tiles", op="batch", kind="tiles", jobs=16, sub=6, size=1280, spp=16, bounces=24, p=0.8, k=16),
        # the gradient of a full-size inverse-rendering step
        dict(name="adjoint_512", op="adjoint", grid=64, size=512, spp=32, bounces=4, p=0.8, k=16),
        # one iteration of the inverse-rendering loop at its default size
        dict(name="inverse_step", op="inverse", grid=32, size=128, spp=8, bounces=4, p=0.8, k=16),
        # ray-set queries (picking, visibility, collision)
        dict(name="ray_queries", op="rays", inst=64, sub=6, rays=262144),
        # an edited scene: upload and a preview frame
        dict(name="upload_preview", op="upload", inst=64, sub=7, w=480, h=270, spp=1, bounces=4, p=0.8, k=16),
        # the tone map of a frame loop that owns its device memory
        dict(name="tonemap_hd", op="tonemap", w=1920, h=1080, host=False),
    ]


def draw(rng):
    """One more case of these ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    p = round(rng.uniform(0.5, 0.9), 3)
    op = rng.choice(["render", "render", "render", "render", "batch", "batch", "adjoint", "inverse", "rays", "upload",
                     "tonemap"])
    if op == "render":
        scene = rng.choice(["box", "mixed", "instanced", "instanced"])
        w = log(48, 1920)
        h = max(27, int(w * rng.uniform(0.5, 1.0)))
        spp = min(log(1, 64), max(1, 100_000_000 // (w * h)))
        c = dict(op=op, scene=scene, w=w, h=h, spp=spp, bounces=log(2, 32), p=p, k=rng.choice([4, 8, 16]),
                 host=rng.random() < 0.5, film64=rng.random() < 0.2)
        if scene == "instanced":
            c.update(inst=log(2, 100), sub=rng.choice([4, 5, 6, 7]))
        return c
    if op == "batch":
        kind = rng.choice(["jobs", "tiles"])
        return dict(op=op, kind=kind, jobs=log(3, 24), sub=rng.choice([4, 5, 6]),
                    size=log(64, 320) if kind == "jobs" else log(300, 1600), spp=log(1, 24), bounces=log(4, 32), p=p,
                    k=rng.choice([4, 8, 16]))
    if op == "adjoint":
        return dict(op=op, grid=rng.choice([16, 32, 48, 64]), size=log(96, 512), spp=log(4, 32), bounces=log(2, 8),
                    p=p, k=rng.choice([4, 8, 16]))
    if op == "inverse":
        return dict(op=op, grid=rng.choice([16, 24, 32]), size=log(64, 192), spp=log(2, 16), bounces=log(2, 8), p=p,
                    k=rng.choice([8, 16]))
    if op == "rays":
        return dict(op=op, inst=log(3, 100), sub=rng.choice([4, 5, 6]), rays=log(1000, 700_000))
    if op == "upload":
        w = log(64, 640)
        return dict(op=op, inst=log(2, 100), sub=rng.choice([4, 5, 6, 7]), w=w, h=max(27, int(w * rng.uniform(0.5, 1.0))),
                    spp=log(1, 4), bounces=log(2, 8), p=p, k=rng.choice([4, 8, 16]))
    w = log(96, 3840)
    return dict(op=op, w=w, h=max(27, int(w * rng.uniform(0.4, 1.0))), host=rng.random() < 0.4)


# ---- scenes ----------------------------------------------------------------------

def _cfg(k):
    # 4 hero wavelengths go with 81 bins on 380-780 nm (the box-room configuration), the rest with the default bins
    return SpectralConfig(81, 380.0, 780.0, 4) if k == 4 else SpectralConfig(hero_k=k)


def _camera(pos, look_at, w, h, fov, dof=0.0, f=1.0):
    return Camera(pos, look_at, [0, 0, 1], w, fov, w / (h - 0.5), dof, f)


def _tri_mesh(name, V, N, F):
    V = np.concatenate([np.zeros((1, 3)), V]).astype(np.float32)
    N = np.concatenate([[[0.0, 0.0, 1.0]], N]).astype(np.float32)
    return TriMeshData(name, V, N, np.concatenate([F + 1, F + 1], axis=1).astype(np.uint32))


@functools.lru_cache(maxsize=None)
def _icosphere(sub):
    V, N, F = synth.displaced_icosphere(sub, 1234)
    return _tri_mesh("icosphere%d" % sub, V, N, F)


@functools.lru_cache(maxsize=None)
def _uv_sphere():
    return _tri_mesh("uvsphere", *synth.uv_sphere())


@functools.lru_cache(maxsize=None)
def _quad(lo, hi):
    # one unit off the plane of the loader's dummy vertex; the object transform moves it back
    V = np.array([[lo, lo, 1], [hi, lo, 1], [hi, hi, 1], [lo, hi, 1]], np.float64)
    return _tri_mesh("quad", V, np.tile([[0.0, 0.0, 1.0]], (4, 1)), np.array([[0, 1, 2], [0, 2, 3]]))


def _wavelengths(cfg):
    return np.linspace(float(cfg.inf), float(cfg.sup), cfg.n_bins)


def _smooth(rng, cfg, lo, hi):
    lam = _wavelengths(cfg)
    v = sum(rng.uniform(0.2, 1.0) * np.exp(-0.5 * ((lam - rng.uniform(380, 780)) / rng.uniform(30, 120)) ** 2)
            for _ in range(3))
    v = (v - v.min()) / max(v.max() - v.min(), 1e-6)
    a = rng.uniform(lo, hi - 0.1)
    return (a + (rng.uniform(a + 0.1, hi) - a) * v).astype(np.float32)


def _flat(cfg, x):
    return np.full(cfg.n_bins, x, np.float32)


def _blackbody(cfg, T, peak):
    return (synth.planck(_wavelengths(cfg), T) / synth.planck([560.0], T)[0] * peak).astype(np.float32)


def _material(rng, cfg, name):
    kind = ["lambertian", "blinn", "thinfilm"][int(rng.integers(0, 3))]
    # an even exponent keeps powf defined for back-facing half vectors
    alpha = np.float32(2 * int(round(np.exp(rng.uniform(np.log(8), np.log(2048))) / 2)))
    if kind == "lambertian":
        return Material(kind, name, albedo=_smooth(rng, cfg, 0.05, 0.9))
    if kind == "blinn":
        m = Material(kind, name, Kd=_smooth(rng, cfg, 0.05, 0.6), Ks=_flat(cfg, rng.uniform(0.2, 0.5)),
                     Kt=_flat(cfg, 0.0), Le=_flat(cfg, 0.0), ior=_flat(cfg, 1.54), alpha=alpha)
        blinn_init(m, cfg)
        return m
    return Material(kind, name, film_ior=_flat(cfg, rng.uniform(1.33, 1.6)), base_ior=_flat(cfg, 1.5), alpha=alpha,
                    d=np.float32(rng.uniform(200, 800)))


def _place(s, degrees, t):
    return Transform.scale([s, s, s]).then(Transform.rotate([0, 0, 1], degrees)).then(Transform.translate(t))


def _quad_light(sc, name, scale, pos, rad):
    T = Transform.scale([scale, scale, 1]).then(Transform.rotate([1, 0, 0], 180)).then(Transform.translate(pos))
    sc.materials.append(Material("diremitter", "emitter_" + name, radiance=rad, specular=np.float32(2)))
    sc.objects.append(Object("plane", name, T, len(sc.materials) - 1, len(sc.objects)))
    c0, c1 = (np.linalg.norm(T.column(k)) for k in (0, 1))
    sc.lights.append(LightDef("quaddir", name, radiance=rad, inv_area=np.float32(1.0 / (c0 * c1)), spec=np.float32(2),
                              T=T, obj=len(sc.objects) - 1))


def _mesh_object(sc, mesh, T, mat):
    if mesh not in sc.meshes:
        sc.meshes.append(mesh)
    sc.objects.append(Object("trimesh", "o%d" % len(sc.objects), T, mat, len(sc.objects), sc.meshes.index(mesh)))


def _instanced(rng, inst, sub, w, h, k):
    cfg = _cfg(k)
    sc = SceneData(cfg)
    side = int(np.ceil(np.sqrt(inst)))
    extent = side * 1.1
    sc.cam = _camera([0.0, -0.95 * extent, 0.75 * extent], [0, 0, 0.2], w, h, 50)
    sc.materials.append(Material("lambertian", "ground", albedo=_flat(cfg, 0.5)))
    _mesh_object(sc, _quad(-1, 1), Transform.scale([12, 12, 1]).then(Transform.translate([0, 0, -1])), 0)
    for i in range(inst):
        sc.materials.append(_material(rng, cfg, "m%d" % i))
        at = [(i % side - (side - 1) / 2) * 1.1, (i // side - (side - 1) / 2) * 1.1, 0.45]
        _mesh_object(sc, _icosphere(sub), _place(0.45, rng.uniform(0, 360), at), len(sc.materials) - 1)
    _quad_light(sc, "key", 1.5, [-2.0, -1.0, 6.0], _blackbody(cfg, 6500.0, 3.0))
    _quad_light(sc, "fill", 1.0, [3.0, 2.0, 5.0], _blackbody(cfg, 4000.0, 2.0))
    return sc


def _box(rng, w, h, k):
    with tempfile.TemporaryDirectory() as d:
        sc = load_nls(synth.box_room(d, width=64, light_peak=float(rng.uniform(4.0, 8.0))), _cfg(k))
    sc.cam = _camera([0.5, -1.4, 0.5], [0.5, 0.5, 0.5], w, h, 40)
    return sc


def _mixed(rng, w, h, k):
    lights = ["sphere", "quaddir", "point", "direction", "ambient"]
    with tempfile.TemporaryDirectory() as d:
        sc = load_nls(synth.mixed(d, lights=lights, seed=int(rng.integers(1 << 30)), subdiv=4), _cfg(k))
    sc.cam = _camera([0.0, -6.0, 2.2], [0.0, 0.0, 0.8], w, h, 45, dof=0.1, f=6.0)
    return sc


def _filled_box(rng, sub, w, h, k):
    """The box room with 1 to 32 instances standing on its floor."""
    sc = _box(rng, w, h, k)
    inst = int(rng.integers(1, 33))
    side = int(np.ceil(np.sqrt(inst)))
    spacing = 0.9 / side
    for i in range(inst):
        sc.materials.append(_material(rng, sc.cfg, "m%d" % i))
        at = [0.05 + (i % side + 0.5) * spacing, 0.05 + (i // side + 0.5) * spacing, 0.4 * spacing]
        _mesh_object(sc, _icosphere(sub), _place(0.4 * spacing, rng.uniform(0, 360), at), len(sc.materials) - 1)
    return sc


@functools.lru_cache(maxsize=None)
def _tiles(grid):
    s = 8.0 / grid
    return [Transform.scale([s, s, 1]).then(Transform.translate([-4.0 + j * s, -4.0 + i * s, -1.0]))
            for i in range(grid) for j in range(grid)]


def _diff(rng, grid, size, k):
    """A ground of grid x grid thin-film tiles under 64 Lambertian spheres."""
    cfg = _cfg(k)
    sc = SceneData(cfg)
    sc.cam = _camera([0.0, -7.5, 8.5], [0.0, -0.3, 0.0], size, size, 45)
    film, base = _flat(cfg, 1.45), _flat(cfg, 1.6)
    for i, T in enumerate(_tiles(grid)):
        sc.materials.append(Material("thinfilm", "film%d" % i, film_ior=film, base_ior=base, alpha=np.float32(8),
                                     d=np.float32(rng.uniform(200, 800))))
        _mesh_object(sc, _quad(0, 1), T, i)
    for i in range(64):
        sc.materials.append(Material("lambertian", "alb%d" % i, albedo=_smooth(rng, cfg, 0.1, 0.9)))
        r = 0.22 + 0.08 * float(rng.uniform())
        _mesh_object(sc, _uv_sphere(), _place(r, 0.0, [i % 8 - 3.5, i // 8 - 3.5, r + 0.05]), len(sc.materials) - 1)
    _quad_light(sc, "key", 3.0, [0.0, 3.0, 7.0], _blackbody(cfg, 6500.0, 4.0))
    _quad_light(sc, "fill", 2.0, [2.5, 5.0, 6.0], _blackbody(cfg, 3500.0, 2.5))
    return sc


def _scene(case, rng):
    if case.get("scene") == "box":
        return _box(rng, case["w"], case["h"], case["k"])
    if case.get("scene") == "mixed":
        return _mixed(rng, case["w"], case["h"], case["k"])
    return _instanced(rng, case["inst"], case["sub"], case["w"], case["h"], case["k"])


# ---- prepare and run ---------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    st = {"case": case, "seed": int(seed)}
    op = case["op"]
    if op == "tonemap":
        h, w = case["h"], case["w"]
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        # linear radiance: a smooth field over two decades with noise
        y = torch.linspace(0, 3, h, device="cuda")[:, None, None]
        x = torch.linspace(0, 5, w, device="cuda")[None, :, None]
        ch = torch.rand(3, generator=g, device="cuda") * 6
        img = torch.exp(1.5 * torch.sin(y + x + ch) - 1.0) * (0.5 + torch.rand(h, w, 3, generator=g, device="cuda"))
        img = img.float().contiguous()
        if case["host"]:
            st.update(ctx=Context(0), img=img.cpu().numpy())
        else:
            st.update(img=img, tm=torch.empty_like(img), b=torch.empty(img.shape, dtype=torch.uint8, device="cuda"))
        return st
    ctx = st["ctx"] = Context(0)
    if op == "render":
        ctx.upload(FlatScene(_scene(case, rng)))
        st["settings"] = (case["spp"], case["bounces"], case["p"])
        st["flags"] = L.FLAG_FP64_FILM if case["film64"] else 0
        if not case["host"]:
            st["out"] = torch.empty(case["h"], case["w"], 3, dtype=torch.float64 if case["film64"] else torch.float32,
                                    device="cuda")
    elif op == "batch":
        n, size, spp = case["jobs"], case["size"], case["spp"]
        if case["kind"] == "jobs":
            scenes, jobs = [], []
            # the jobs' sizes belong to the case, not to the seed
            sizes = np.random.default_rng([n, size, spp])
            for k in range(n):
                w = max(16, int(size * sizes.uniform(0.5, 1.0)))
                scenes.append(_filled_box(rng, case["sub"], w, w, case["k"]))
                jobs.append(dict(scene=k, spp=max(1, int(spp * sizes.uniform(0.5, 1.0))),
                                 max_scatterings=case["bounces"], sample_p=case["p"], seed=int(seed) + k))
            ctx.upload_many(scenes)
            outs = [torch.zeros(w, w, 3, device="cuda") for w in (s.cam.width for s in scenes)]
            st.update(outs=outs, ret=outs)
        else:
            w, h = size, int(size * 9 / 16)
            ctx.upload_many([_instanced(rng, 16, case["sub"], w, h, case["k"])])
            nx = int(math.ceil(math.sqrt(n)))
            ny = int(math.ceil(n / nx))
            xs, ys = ([round(i * m / q) for i in range(q + 1)] for m, q in ((w, nx), (h, ny)))
            jobs = [dict(scene=0, spp=spp, max_scatterings=case["bounces"], sample_p=case["p"], seed=int(seed),
                         rect=(xs[i], ys[j], xs[i + 1] - xs[i], ys[j + 1] - ys[j]))
                    for j in range(ny) for i in range(nx)]
            out = torch.zeros(h, w, 3, device="cuda")
            st.update(outs=[out] * len(jobs), ret=[out])
        st.update(jobs=jobs, ptrs=[o.data_ptr() for o in st["outs"]])
    elif op in ("adjoint", "inverse"):
        flat = st["flat"] = ctx.upload(FlatScene(_diff(rng, case["grid"], case["size"], case["k"])))
        st["settings"] = (case["spp"], case["bounces"], case["p"])
        shape = (case["size"], case["size"], 3)
        if op == "adjoint":
            d = torch.from_numpy(rng.normal(size=shape).astype(np.float32)).cuda()
            gs = torch.empty(int(flat.scene.n_spectra), int(flat.scene.spec.n_bins), device="cuda")
            gm = torch.empty(int(flat.scene.n_materials), 4, device="cuda")
            st.update(d=d, gs=gs, gm=gm, img=torch.empty(shape, device="cuda"))
        else:
            st["target"] = rng.uniform(0.0, 1.0, shape).astype(np.float32)
    elif op == "rays":
        sc = _instanced(rng, case["inst"], case["sub"], 64, 36, 16)
        ctx.upload(FlatScene(sc))
        n, ext = case["rays"], 0.55 * np.ceil(np.sqrt(case["inst"]))
        # half from the camera towards the instances, half from among them in all directions
        a = n // 2
        o = rng.uniform([-ext, -ext, 0.05], [ext, ext, 1.2], (n, 3))
        o[:a] = np.array(sc.cam.pos, np.float64)
        t = rng.uniform([-ext, -ext, 0.0], [ext, ext, 1.0], (n, 3))
        u = t - o
        u[a:] = rng.normal(size=(n - a, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        st["rays"] = np.concatenate([o, u], axis=1).astype(np.float32)
        # shadow rays towards points of the key light
        q = np.array([-2.0, -1.0, 6.0]) + rng.uniform(-1.5, 1.5, (n, 3)) * [1, 1, 0]
        d = q - o
        dist = np.linalg.norm(d, axis=1)
        st["shadow"] = np.concatenate([o, d / dist[:, None]], axis=1).astype(np.float32)
        st["tmax"] = dist.astype(np.float32)
        st["skip"] = np.uint32(sc.lights[0].obj)
    elif op == "upload":
        st["flat"] = FlatScene(_instanced(rng, case["inst"], case["sub"], case["w"], case["h"], case["k"]))
        st["settings"] = (case["spp"], case["bounces"], case["p"])
    return st


def run(st):
    case, seed, op = st["case"], st["seed"], st["case"]["op"]
    if op == "tonemap":
        img = st["img"]
        if case["host"]:
            return st["ctx"].tonemap(img, 0.12)
        rc = L.lib().lgpu_tonemap_noalloc(img.data_ptr(), case["w"], case["h"], 0.12, st["tm"].data_ptr(),
                                          st["b"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        L.check(None, rc, "tonemap_noalloc")
        return st["tm"], st["b"]
    ctx = st["ctx"]
    if op == "render":
        if case["host"]:
            return ctx.render(*st["settings"], seed=seed, flags=st["flags"])
        ctx.render_device(*st["settings"], st["out"].data_ptr(), seed=seed, flags=st["flags"],
                          stream=torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if op == "batch":
        ctx.render_batch_device(st["jobs"], st["ptrs"], stream=torch.cuda.current_stream().cuda_stream)
        return st["ret"]
    if op == "adjoint":
        ctx.adjoint_device(*st["settings"], st["d"].data_ptr(), st["gs"].data_ptr(), st["gm"].data_ptr(),
                           st["img"].data_ptr(), seed=seed, stream=torch.cuda.current_stream().cuda_stream)
        return st["img"], st["gs"], st["gm"]
    if op == "inverse":
        ctx.update_materials(st["flat"])
        img = ctx.render(*st["settings"], seed=seed)
        d = (img - st["target"]) * np.float32(2.0 / img.size)
        gs, gm = ctx.adjoint(*st["settings"], d, seed=seed + 0x9E3779B9)
        return img, gs, gm
    if op == "rays":
        h = ctx.trace(st["rays"])
        occ = ctx.trace_any(st["shadow"], st["tmax"], st["skip"])
        return {**{f: np.ascontiguousarray(h[f]).astype(np.int64 if h[f].dtype.kind == "u" else h[f].dtype)
                   for f in h.dtype.names}, "occluded": occ.astype(np.uint8)}
    ctx.upload(st["flat"])
    return ctx.render(*st["settings"], seed=seed)


# ---- what a pass cannot do without -------------------------------------------------

# FP32 operations of one ray through an 8-wide tree over a scene (9 node tests, 3 triangle tests, 1.5 instance
# entries) and of one shading vertex per hero wavelength and in all
RAY_FLOPS, HERO_FLOPS, VERTEX_FLOPS = 1500, 40, 300


def _mesh_bytes(sub):
    # leaf triangles, shading records and 8-wide nodes of one icosphere, each read once
    return 20 * 4 ** sub * (36 + 48 + 28)


def work(case):
    op = case["op"]
    if op == "tonemap":
        n = case["w"] * case["h"]
        return {"bytes": n * (12 + 12 + 3), "flops": 3 * n * 30}
    if op == "rays":
        # 24 B in and 48 B out per closest-hit ray, 32 in and 1 out per shadow ray
        return {"bytes": case["rays"] * (24 + 48 + 32 + 1) + _mesh_bytes(case["sub"]),
                "flops": 2 * case["rays"] * RAY_FLOPS}
    p, b, k = case["p"], case["bounces"], case["k"]
    # scattering vertices of a path that always hits: Russian roulette with probability p, at most b + 1
    vertices = (1 - p ** (b + 1)) / (1 - p)
    if op == "batch":
        frac = 0.75 if case["kind"] == "jobs" else 1.0
        pix = case["jobs"] * (0.75 * case["size"]) ** 2 if case["kind"] == "jobs" else case["size"] ** 2 * 9 / 16
        paths = pix * max(1, frac * case["spp"])
    else:
        pix = case["w"] * case["h"] if "w" in case else case["size"] ** 2
        paths = pix * case["spp"]
    passes = {"adjoint": 2, "inverse": 3}.get(op, 1)
    flops = passes * paths * vertices * 0.6 * (2 * RAY_FLOPS + VERTEX_FLOPS + k * HERO_FLOPS)
    scene = _mesh_bytes(case["sub"]) if "sub" in case else 100_000
    return {"bytes": pix * 12 * passes + scene * (2 if op == "upload" else 1), "flops": flops}


def exact(case, seed):
    """The tone map in double precision; None for the rest: a path's random
    decisions and a ray's nearest face are not numbers that another precision
    approximates."""
    if case["op"] != "tonemap":
        return None
    img = prepare(dict(case, host=False), seed)["img"].double()
    lum = 0.2126 * img[..., 0] + 0.7152 * img[..., 1] + 0.0722 * img[..., 2]
    x = 10.0 * img * (0.12 / torch.exp(torch.log(lum.clamp_min(2.0 ** -23)).mean()))
    tm = x * (0.3 * x + 0.14) / (x * (0.3 * x + 2.8) + 10.0)
    return (tm.cpu().numpy() if case["host"] else tm), None
