"""The measured cases: what a user of this framework has it do, through its
public entry points.

A case names a kind and its sizes:
  render   PerPixelRenderer.render, the film copied to the host: the renderer's
           own estimator on the Cornell box (5 quads, 2 spheres) or on the
           displaced icosphere (20 x 4^levels triangles, plane, sky, area
           light), the physical estimator on two rooms joined by a door (a
           mesh of 2 x quads^2 triangles) or on an instanced terrain (a
           two-level tree)
  guided   render_guided on the two rooms with a network that no longer trains
  batch    several seeded scenes rendered in one call, by shared wavefronts
           under CUDA graphs ("fused") or on concurrent streams
  mlt      MetropolisRenderer.render
  trace    closest or any hit of a batch of rays, from host arrays
           (GpuScene.intersect / occluded) or device buffers
           (gbrt_trace_closest_device / gbrt_trace_any_device)
  eval     Guide.eval, train: Guide.train_step on a resumed checkpoint

Every seed turns the meshes, moves the spheres and the camera and draws other
samples. Meshes are cached before they are turned; nothing else is.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import renderer_gb300 as rg
from renderer_gb300 import Context, GpuScene, PerPixelRenderer, _abi, workloads
from renderer_gb300.batch import BatchJob, render_batch, render_batch_fused
from renderer_gb300.chains import MetropolisRenderer
from renderer_gb300.guiding import Guide, guide_params, render_guided, scene_bounds
from renderer_gb300.runtime import HIT_DTYPE, make_rays
from renderer_gb300.scene import SceneData, render_params


# --------------------------------------------------------------- the cases --
def listed():
    return [
        # Smallest call: a thumbnail while a user edits a scene; one sample a
        # pixel, odd size, the renderer's default depth. Latency and launches.
        {"name": "preview", "kind": "render", "scene": "cornell", "width": 67, "height": 45, "xs": 1, "ys": 1,
         "depth": 5},
        # The Cornell box of the benchmark: tiny tree, closed room, so shading
        # and the path state dominate.
        {"name": "cornell", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "xs": 4, "ys": 4,
         "depth": 8},
        # The headline frame: 1.31M triangles, 67M paths.
        {"name": "icosphere", "kind": "render", "scene": "icosphere", "levels": 8, "width": 1024, "height": 1024,
         "xs": 8, "ys": 8, "depth": 12},
        # Physical estimator, indirect light, 500,000 triangles, a few samples.
        {"name": "rooms", "kind": "render", "scene": "rooms", "quads": 500, "width": 1024, "height": 768, "xs": 4,
         "ys": 1, "depth": 12},
        # One view of an instanced landscape: two-level tree, sampled sky.
        {"name": "terrain", "kind": "render", "scene": "terrain", "quads": 700, "width": 1920, "height": 1080, "xs": 1,
         "ys": 1, "depth": 16},
        # A pass with a trained guide: inference of every vertex's mixture.
        {"name": "guided", "kind": "guided", "quads": 300, "width": 1024, "height": 768, "spp": 2, "passes": 2,
         "depth": 12},
        # Many small images in shared wavefronts.
        {"name": "batch", "kind": "batch", "how": "fused", "jobs": 10, "quads": 120, "res": 200, "xs": 4, "ys": 4,
         "depth": 8},
        # Markov chains with the renderer's default options.
        {"name": "metropolis", "kind": "mlt", "width": 256, "height": 256, "mutations": 16, "depth": 5},
        # A host program's own rays, a few thousand at a time.
        {"name": "rays_host", "kind": "trace", "scene": "icosphere", "levels": 3, "rays": 5003, "any": False,
         "device": False},
        # A device program's rays: camera and bounce rays into the large mesh.
        {"name": "rays_closest", "kind": "trace", "scene": "icosphere", "levels": 8, "rays": 4000037, "any": False,
         "device": True},
        # Guide inference on a program's own points.
        {"name": "guide_eval", "kind": "eval", "rows": 200003},
        # One optimizer step on the samples of a pass, 2^18 as configured.
        {"name": "guide_train", "kind": "train", "rows": 262144},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case. Image sides, samples, rays and rows are log-uniform and
    mostly odd; meshes have 20 x 4^3 .. 20 x 4^8 or 2 x 40^2 .. 2 x 700^2
    triangles; at most 2^24 paths, four million rays or a million rows."""
    kind = rng.choice(["render", "render", "render", "render", "guided", "batch", "mlt", "trace", "trace", "eval",
                       "train"])
    if kind in ("render", "guided"):
        c = {"kind": kind, "width": _log(rng, 24, 1600), "height": _log(rng, 24, 1200),
             "depth": rng.randint(3, 16)}
        room = max(1, (1 << 24) // (c["width"] * c["height"]))
        if kind == "guided":
            c.update(quads=_log(rng, 40, 500), spp=min(rng.randint(1, 4), room), passes=rng.randint(1, 3))
            return c
        spp = min(_log(rng, 1, 64), room)
        c["xs"] = rng.randint(1, max(1, int(math.sqrt(spp))))
        c["ys"] = max(1, spp // c["xs"])
        c["scene"] = rng.choice(["cornell", "icosphere", "rooms", "terrain"])
        if c["scene"] == "icosphere":
            c["levels"] = rng.randint(3, 8)
        elif c["scene"] != "cornell":
            c["quads"] = _log(rng, 40, 700)
        return c
    if kind == "batch":
        return {"kind": kind, "how": rng.choice(["fused", "streams"]), "jobs": rng.randint(2, 16),
                "quads": _log(rng, 40, 200), "res": _log(rng, 32, 300), "xs": rng.randint(1, 4),
                "ys": rng.randint(1, 4), "depth": rng.randint(3, 10)}
    if kind == "mlt":
        return {"kind": kind, "width": _log(rng, 48, 400), "height": _log(rng, 48, 400),
                "mutations": rng.randint(4, 24), "depth": rng.randint(3, 8)}
    if kind == "trace":
        c = {"kind": kind, "scene": rng.choice(["cornell", "icosphere", "rooms", "terrain"]),
             "rays": _log(rng, 100, 4000000), "any": rng.random() < 0.5, "device": rng.random() < 0.5}
        if c["scene"] == "icosphere":
            c["levels"] = rng.randint(3, 8)
        elif c["scene"] != "cornell":
            c["quads"] = _log(rng, 40, 700)
        if not c["device"]:
            c["rays"] = min(c["rays"], 400003)
        return c
    return {"kind": kind, "rows": _log(rng, 100, 1000000)}


# ------------------------------------------------------------------ scenes --
@functools.lru_cache(maxsize=None)
def _icosphere(levels):
    return workloads.displaced_icosphere(levels, 0, 0.1, True)


@functools.lru_cache(maxsize=None)
def _grid(quads, x0, x1, y0, y1, z, depth, seed):
    return workloads.displaced_grid(quads, x0, x1, y0, y1, z, depth, seed)


@functools.lru_cache(maxsize=None)
def _terrain(quads):
    return workloads.terrain(2 * quads, quads, 8.0, 4.0, 0.8, 0)


@functools.lru_cache(maxsize=None)
def _sky(width, height):
    return workloads.synthetic_sky(width, height, 0)[0]


def _turned(xyz, angle, axis=1):
    """xyz (N, 9) turned about a coordinate axis."""
    a, b = [k for k in range(3) if k != axis]
    c, s = np.float32(math.cos(angle)), np.float32(math.sin(angle))
    p = xyz.reshape(-1, 3)
    q = p.copy()
    q[:, a] = c * p[:, a] + s * p[:, b]
    q[:, b] = c * p[:, b] - s * p[:, a]
    return q.reshape(-1, 9)


def _scene(case, seed):
    """The SceneData of a case: the workloads' scenes with the seed's pose."""
    rng = np.random.default_rng([int(seed), 17])
    w, h = case.get("width", 64), case.get("height", 64)
    kind = case.get("scene", "rooms")
    if kind == "cornell":
        s = workloads.cornell_box(w, h)
        s.spheres = [((-0.45 + rng.uniform(-0.1, 0.1), 0.35, -0.3), 0.35, s.spheres[0][2]),
                     ((0.45 + rng.uniform(-0.1, 0.1), 0.35, 0.25), 0.35, s.spheres[1][2])]
        eye = (rng.uniform(-0.1, 0.1), 1.0 + rng.uniform(-0.1, 0.1), 3.4)
    elif kind == "icosphere":
        s = workloads.icosphere_scene(levels=1, width=w, height=h, env_size=(16, 8))
        pos, nrm = _icosphere(case["levels"])
        a = rng.uniform(0, 2 * math.pi)
        s.tri_pos, s.tri_nrm = _turned(pos, a), _turned(nrm, a)
        s.tri_mat = np.zeros(len(pos), np.int32)
        s.env = _sky(1024, 512)
        eye = (rng.uniform(-0.2, 0.2), 0.4 + rng.uniform(-0.1, 0.1), 3.2)
    elif kind == "rooms":
        s = workloads.two_rooms(w, h, mesh_quads=2)
        n = case["quads"]
        pos, nrm = _grid(n, 0.6, 3.4, 0.2, 2.6, 2.97, 0.3, 0)
        p = pos.reshape(-1, 3).copy()
        p[:, 0] += np.float32(rng.uniform(-0.1, 0.1))
        s.tri_pos, s.tri_nrm = p.reshape(-1, 9), nrm
        s.tri_mat = np.full(len(pos), s.tri_mat[0], np.int32)
        eye = (0.4 + rng.uniform(-0.1, 0.1), 1.5, 0.6 + rng.uniform(-0.1, 0.1))
    else:
        s, _ = workloads.terrain_instances(seed=int(seed) & 0xffff, nx=2, nz=2, width=w, height=h, env_size=(16, 8),
                                           views=1)
        pos, nrm = _terrain(case["quads"])
        s.meshes[0].update(pos=pos, nrm=nrm, mat=np.zeros(len(pos), np.int32))
        s.env = _sky(2048, 1024)
        eye = s.camera["eye"]
    s.camera = dict(s.camera, eye=tuple(float(x) for x in eye))
    return s


def _batch_job(case, seed, i):
    """A small scene in the manner of workloads.batch_scene: a diffuse box, a
    turned relief, spheres and one or two area lights."""
    rng = np.random.default_rng([int(seed), 23, i])
    s = SceneData()
    s.flags = _abi.SCENE_GPU_BUILD
    wall = s.add_material(_abi.MAT_DIFFUSE, kd=tuple(rng.uniform(0.5, 0.8, 3)))
    mats = [s.add_material(_abi.MAT_DIFFUSE, kd=tuple(rng.uniform(0.2, 0.85, 3))),
            s.add_material(_abi.MAT_MIRROR), s.add_material(_abi.MAT_TRANSPARENT, ior=1.5),
            s.add_material(_abi.MAT_BLINN, kd=(0.3, 0.3, 0.3), ks=(0.5, 0.5, 0.5),
                           exponent=float(rng.uniform(10.0, 500.0)))]
    s.quads = [((-2, 0, -2), (2, 0, -2), (2, 0, 2), (-2, 0, 2), wall),
               ((-2, 3, -2), (-2, 3, 2), (2, 3, 2), (2, 3, -2), wall),
               ((-2, 0, -2), (-2, 3, -2), (2, 3, -2), (2, 0, -2), wall),
               ((-2, 0, -2), (-2, 0, 2), (-2, 3, 2), (-2, 3, -2), wall),
               ((2, 0, -2), (2, 3, -2), (2, 3, 2), (2, 0, 2), wall)]
    pos, nrm = _grid(case["quads"] + 7 * (i % 4), -1.0, 1.0, -1.0, 1.0, 0.0, 0.15, i % 4)
    a = rng.uniform(0, 2 * math.pi)
    s.tri_pos = _turned(pos, a).reshape(-1, 3)
    s.tri_pos = (s.tri_pos + np.array([0.0, 1.2, 0.0], np.float32)).reshape(-1, 9)
    s.tri_nrm = _turned(nrm, a)
    s.tri_mat = np.full(len(pos), mats[i % 4], np.int32)
    for _ in range(int(rng.integers(2, 6))):
        r = float(rng.uniform(0.1, 0.45))
        s.spheres.append(((rng.uniform(-1.5, 1.5), rng.uniform(r, 2.5), rng.uniform(-1.5, 1.5)), r,
                          mats[int(rng.integers(4))]))
    for _ in range(int(rng.integers(1, 3))):
        e = float(rng.uniform(5.0, 50.0))
        s.lights.append(dict(type=_abi.LIGHT_AREA, origin=(rng.uniform(-1.5, 1), 2.99, rng.uniform(-1.5, 1)),
                             u=(0.5, 0, 0), v=(0, 0, 0.5), intensity=(e, e, e)))
    res = case["res"] + 16 * (i % 5)  # images of uneven size
    s.camera = dict(eye=(rng.uniform(-0.5, 0.5), 1.5, 6.5), look_at=(0, 1.5, 0), up=(0, 1, 0),
                    fov=workloads.FOV_40, width=res, height=res - 3)
    return s, render_params(case["xs"], case["ys"], 0.5, case["depth"], seed=int(seed) + i)


def _rays(case, seed):
    """Half the rays as a camera would send them, half as bounces leave the
    surfaces: origins in the scene, directions all around."""
    rng = np.random.default_rng([int(seed), 29])
    s = _scene(case, seed)
    n = case["rays"]
    k = n // 2
    eye, look = np.asarray(s.camera["eye"], np.float32), np.asarray(s.camera["look_at"], np.float32)
    t = np.linspace(0, 1, max(1, k), dtype=np.float32)
    fan = np.stack([0.7 * np.sin(811 * t), 1.2 * (t - 0.5), 0.7 * np.cos(811 * t)], 1).astype(np.float32)
    d0 = (look - eye) + fan[:k]
    org = np.empty((n, 3), np.float32)
    org[:k] = eye
    mid = {"cornell": (0, 1, 0), "icosphere": (0, 0, 0), "rooms": (2, 1.5, 1.5), "terrain": (0, 1.5, 0)}[case["scene"]]
    half = {"cornell": 0.9, "icosphere": 1.3, "rooms": 1.4, "terrain": 3.0}[case["scene"]]
    org[k:] = np.asarray(mid, np.float32) + half * (2 * rng.random((n - k, 3), np.float32) - 1)
    dirs = np.concatenate([d0, rng.standard_normal((n - k, 3), np.float32)])
    return s, make_rays(org, dirs, tmax=4.0 if case["any"] else np.inf)


_ctx = None


def _context():
    """One context for the whole program, as a user's program keeps one."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


# ------------------------------------------------------------------- guide --
_BOX = np.array([0.0, 0.0, 0.0, 8.0, 3.0, 3.0], np.float32)


def _net_state(seed):
    """A checkpoint in the middle of training: uniform weights of the
    network's own initial size, moments of gradients about 1e-2."""
    rng = np.random.default_rng([int(seed), 31])
    parts = [rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / b) * s
             for (a, b), s in zip(((64, 208), (64, 64), (64, 64), (40, 64)), (1, 1, 1, 0.4))]
    w = np.concatenate(parts).astype(np.float32)
    return {"params": w, "adam_m": (1e-3 * rng.standard_normal(len(w))).astype(np.float32),
            "adam_v": (1e-4 * rng.uniform(0.5, 2.0, len(w))).astype(np.float32), "step": 512}


def _unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _points(rows, seed, sampled):
    """Points in the rooms, normals and outgoing directions; with `sampled`
    an incident direction and the weight of a radiance sample as well."""
    rng = np.random.default_rng([int(seed), 37])
    p = _BOX[:3] + rng.random((rows, 3), np.float32) * (_BOX[3:] - _BOX[:3])
    cols = [p, _unit(rng.standard_normal((rows, 3), np.float32)), _unit(rng.standard_normal((rows, 3), np.float32))]
    if sampled:
        cols += [_unit(rng.standard_normal((rows, 3), np.float32)), rng.exponential(1.0, (rows, 1))]
    return np.concatenate(cols, 1).astype(np.float32)


# ------------------------------------------------------------ prepare, run --
def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    st = {"kind": kind, "ctx": ctx}
    if kind in ("render", "guided", "mlt"):
        s = _scene(dict(case, scene="cornell") if kind == "mlt" else case, seed)
        st["scene"] = scene = GpuScene(ctx, s)
        cam = s.camera_struct()
        if kind == "render":
            physical = case["scene"] in ("rooms", "terrain")
            r = PerPixelRenderer(scene, cam, {"pt-x-samples": case["xs"], "pt-y-samples": case["ys"]}, seed=seed,
                                 max_depth=case["depth"])
            if physical:
                r.params.semantics = _abi.SEM_PHYSICAL
            st["renderer"] = r
        elif kind == "mlt":
            st["renderer"] = MetropolisRenderer(scene, cam, {"met-mutations": case["mutations"]}, seed=seed,
                                                max_depth=case["depth"])
        else:
            st["camera"] = cam
            st["params"] = render_params(case["spp"], 1, 0.5, case["depth"], seed, semantics=_abi.SEM_PHYSICAL)
            st["guide"] = Guide(ctx, scene_bounds(scene), seed=1)
            st["guide"].set_weights(_net_state(seed)["params"])
            st["gp"] = guide_params(passes=case["passes"])
    elif kind == "batch":
        made = [_batch_job(case, seed, i) for i in range(case["jobs"])]
        st["how"] = case["how"]
        st["scenes"] = [GpuScene(ctx, s) for s, _ in made]
        st["jobs"] = [BatchJob(g, s.camera_struct(), p) for g, (s, p) in zip(st["scenes"], made)]
    elif kind == "trace":
        s, rays = _rays(case, seed)
        st["scene"] = GpuScene(ctx, s)
        st["any"], st["device"], st["n"] = case["any"], case["device"], len(rays)
        if case["device"]:
            st["rays"] = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
            st["out"] = torch.empty(len(rays), dtype=torch.uint8, device="cuda") if case["any"] else \
                torch.empty((len(rays), 4), dtype=torch.float32, device="cuda")
        else:
            st["rays"] = rays
    else:
        st["guide"] = Guide(ctx, _BOX, seed=1)
        st["guide"].set_state(_net_state(seed))
        st["rows"] = _points(case["rows"], seed, kind == "train")
    return st


def _hits(h):
    """Hit records as their columns (of a device buffer as views: the rays are
    traced on the context's stream, not torch's)."""
    if isinstance(h, torch.Tensor):
        return {"t": h[:, 0], "prim": h.view(torch.int32)[:, 1], "u": h[:, 2], "v": h[:, 3]}
    return {k: h[k] for k in HIT_DTYPE.names}


def run(st):
    kind = st["kind"]
    if kind in ("render", "mlt"):
        return st["renderer"].render()
    if kind == "guided":
        return render_guided(st["scene"], st["camera"], st["params"], st["guide"], st["gp"])[0]
    if kind == "batch":
        return (render_batch_fused if st["how"] == "fused" else render_batch)(st["ctx"], st["jobs"])[0]
    if kind == "trace":
        if not st["device"]:
            return st["scene"].occluded(st["rays"]) if st["any"] else _hits(st["scene"].intersect(st["rays"]))
        rays, out = C.c_void_p(st["rays"].data_ptr()), C.c_void_p(st["out"].data_ptr())
        if st["any"]:
            rg.check(rg.lib().gbrt_trace_any_device(st["scene"].handle, rays, None, st["n"], out, None), st["ctx"].handle)
            return st["out"]
        rg.check(rg.lib().gbrt_trace_closest_device(st["scene"].handle, rays, st["n"], out, None), st["ctx"].handle)
        return _hits(st["out"])
    if kind == "eval":
        return st["guide"].eval(st["rows"])
    loss = st["guide"].train_step(st["rows"], 1e-2)
    now = st["guide"].get_state()
    return {"loss": loss, "params": now["params"], "adam_m": now["adam_m"], "adam_v": now["adam_v"]}


# -------------------------------------------------------------------- work --
_MACS = 24064  # weights of the guide's network


def _triangles(case):
    kind = case.get("scene", "rooms")
    if kind == "cornell":
        return 14
    if kind == "icosphere":
        return 20 * 4 ** case["levels"]
    return (4 if kind == "terrain" else 2) * case["quads"] ** 2


def work(case):
    """Bytes: the scene's positions and normals (72 a triangle) read once, the
    results written once. Flops: 200 a ray for each halving of the triangles
    (a box pair), and about three rays and 500 flops of shading a path; the
    network's products where it runs."""
    kind = case["kind"]
    if kind == "eval":
        return {"bytes": case["rows"] * (36 + 160) + 4 * _MACS, "flops": 2.0 * _MACS * case["rows"]}
    if kind == "train":
        return {"bytes": case["rows"] * 52 + 24 * _MACS, "flops": 6.0 * _MACS * case["rows"]}
    n = _triangles(dict(case, scene="cornell") if kind == "mlt" else case)
    per_ray = 200.0 * math.log2(n + 2)
    if kind == "trace":
        return {"bytes": 72.0 * n + case["rays"] * (33 if case["any"] else 48), "flops": per_ray * case["rays"]}
    if kind == "batch":
        px = sum((case["res"] + 16 * (i % 5)) * (case["res"] + 16 * (i % 5) - 3) for i in range(case["jobs"]))
        return {"bytes": 72.0 * n * case["jobs"] + 12.0 * px,
                "flops": (3 * per_ray + 500) * px * case["xs"] * case["ys"]}
    px = case["width"] * case["height"]
    paths = px * (case["mutations"] if kind == "mlt" else case["spp"] * case["passes"] if kind == "guided"
                  else case["xs"] * case["ys"])
    flops = (3 * per_ray + 500) * paths + (2.0 * 2 * _MACS * paths if kind == "guided" else 0)
    return {"bytes": 72.0 * n + 12.0 * px, "flops": flops}


# ------------------------------------------------------------------- exact --
def _f64(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def _encode(rows):
    """The network's input of (point, normal, outgoing direction) rows."""
    x = _f64(rows[:, :9])
    lo, hi = _f64(_BOX[:3]), _f64(_BOX[3:])
    v = torch.cat([((x[:, :3] - lo) / (hi - lo)).clamp(0, 1), 0.5 * (x[:, 3:6] + 1)], 1)
    a = math.pi * v[:, :, None] * 2.0 ** _f64(np.arange(12))
    bands = torch.stack([torch.sin(a), torch.cos(a)], 3).reshape(len(x), -1)
    mid = (_f64(np.arange(32)) + 0.5) / 32
    th = (torch.acos(x[:, 8].clamp(-1, 1)) / math.pi)[:, None] - mid
    ph = (torch.atan2(x[:, 7], x[:, 6]) / (2 * math.pi) + 0.5)[:, None] - mid
    ph = ph - torch.round(ph)
    return torch.cat([bands, torch.exp(-0.5 * (32 * th) ** 2), torch.exp(-0.5 * (32 * ph) ** 2)], 1)


def _network(w, x):
    o = 0
    for i, (a, b) in enumerate(((64, 208), (64, 64), (64, 64), (40, 64))):
        x = x @ w[o:o + a * b].reshape(a, b).T
        x = torch.relu(x) if i < 3 else x
        o += a * b
    mean = x[:, 8:32].reshape(-1, 8, 3)
    return x[:, :8], mean / torch.linalg.norm(mean, dim=2, keepdim=True), torch.exp(x[:, 32:].clamp(-4, 9))


def _exact_train(case, seed):
    rows, st = _points(case["rows"], seed, True), _net_state(seed)
    w = _f64(st["params"]).requires_grad_(True)
    total = 0.0
    for at in range(0, len(rows), 65536):
        part = rows[at:at + 65536]
        o, mu, k = _network(w, _encode(part))
        wi = _f64(part[:, 9:12])
        c = (mu * wi[:, None]).sum(2)
        lp = torch.log_softmax(o, 1) + torch.log(k / (2 * math.pi)) - torch.log(-torch.expm1(-2 * k)) + k * (c - 1)
        loss = -(_f64(part[:, 12]) * torch.logsumexp(lp, 1)).sum() / len(rows)
        loss.backward()
        total += float(loss.detach())
    g, step = w.grad.cpu().numpy(), st["step"] + 1
    m = 0.9 * st["adam_m"].astype(np.float64) + 0.1 * g
    v = 0.999 * st["adam_v"].astype(np.float64) + 0.001 * g * g
    p = st["params"] - 1e-2 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"loss": total, "params": p, "adam_m": m, "adam_v": v}


def _exact_trace(case, seed):
    """t of every ray against every triangle, the plane and the area light."""
    s, rays = _rays(case, seed)
    o, d = _f64(rays["org"]), _f64(rays["dir"])
    best = torch.full_like(o[:, 0], math.inf)

    def meet(p, e1, e2, square):
        n = torch.linalg.cross(e1, e2)
        det = -(d[:, None] * n).sum(2)
        a = o[:, None] - p
        q = torch.linalg.cross(a, d[:, None].expand_as(a))
        t, u, v = (a * n).sum(2) / det, (q * e2).sum(2) / det, -(q * e1).sum(2) / det
        ok = (u >= 0) & (v >= 0) & (t >= float(np.float32(0.001)))
        ok &= ((u <= 1) & (v <= 1)) if square else (u + v <= 1)
        return torch.where(ok, t, math.inf).min(1).values

    tri = _f64(s.tri_pos).reshape(-1, 3, 3)
    for part in tri.split(256):
        best = torch.minimum(best, meet(part[:, 0], part[:, 1] - part[:, 0], part[:, 2] - part[:, 0], False))
    for L in s.lights:
        if L["type"] == _abi.LIGHT_AREA:
            c = [_f64([L[k]]) for k in ("origin", "u", "v")]
            best = torch.minimum(best, meet(*c, True))
    for p, _ in s.planes:
        p = _f64(np.asarray(p, np.float32))
        t = -((o * p[:3]).sum(1) + p[3]) / (d * p[:3]).sum(1)
        best = torch.minimum(best, torch.where(t >= float(np.float32(0.001)), t, math.inf))
    return {"t": best.cpu().numpy(), "prim": None, "u": None, "v": None}


def exact(case, seed):
    """The network's outputs and its optimizer step, and the hits of small
    batches of rays. None for images: which path a sample takes hangs on
    comparisons in 32 bits, so a pixel has no value in 64 bits that the same
    random numbers lead to."""
    kind = case["kind"]
    if kind == "eval":
        with torch.no_grad():
            w = _f64(_net_state(seed)["params"])
            got = [torch.cat([torch.softmax(o, 1), torch.cat([mu, k[:, :, None]], 2).reshape(-1, 32)], 1)
                   for o, mu, k in (_network(w, _encode(p)) for p in np.array_split(
                       _points(case["rows"], seed, False), 1 + case["rows"] // 65536))]
            return torch.cat(got).cpu()
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "trace" and case["scene"] == "icosphere" and not case["any"] and \
            case["rays"] * _triangles(case) <= 1 << 30:
        return _exact_trace(case, seed)
    return None
