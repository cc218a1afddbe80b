"""The work that users of this package have it do, as cases that can be timed.

Each case goes through the public entry points of fumeng_b200: ray queries on host and on
device buffers, single-view renders from previews to a full-HD frame, batched renders,
one optimisation step over textures (texel update, forward render, adjoint), scene
creation, and post-processing.  Sizes are those of this repository's workloads
(fumeng_b200.synth), tests and benchmark; camera samples per pixel are lowered on the two
largest renders so that a pass stays well under a second.

listed() gives the cases, draw(rng) more of the same ranges, prepare(case, seed) what a
program has in hand before the call, run(state) one pass, work(case) the bytes and
operations a pass cannot do without, exact(case, seed) the same outputs in 64 bits where
they can be had without this package.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import fumeng_b200 as fb
from fumeng_b200 import synth
from fumeng_b200.scene import Mesh, camera_struct

CHAINS = {
    # what a scene file's post-process list names most often
    "display": [(fb.FM_POST_DENOISE, 0.0), (fb.FM_POST_TONEMAP, 1.0), (fb.FM_POST_LINEAR_TO_SRGB, 0.0)],
    "tonemap": [(fb.FM_POST_TONEMAP, 1.2), (fb.FM_POST_LINEAR_TO_SRGB, 0.0)],
}


def listed() -> list:
    return [
        # picking under the cursor in a viewer: few rays, host arrays, latency counts
        {"name": "pick", "kind": "query_host", "mesh": "hit", "rays": 256, "order": "random"},
        # depth pre-pass / lidar sweep from host arrays: coherent rays on the 1.3 M-triangle mesh
        {"name": "primary_host", "kind": "query_host", "mesh": "single", "rays": 129600, "order": "camera"},
        # visibility baking on device buffers: incoherent closest-hit rays, large batch
        {"name": "closest_device", "kind": "query_device", "mesh": "single", "rays": 2000000, "order": "random",
         "any": False},
        # ambient-occlusion style occlusion queries on device buffers, ragged count
        {"name": "occlusion_device", "kind": "query_device", "mesh": "hit", "rays": 1000003, "order": "random",
         "any": True},
        # material preview thumbnail: every BSDF and light kind, a few samples, with AOVs
        {"name": "preview", "kind": "render", "scene": "materials", "width": 64, "height": 64, "spp": 4, "depth": 6,
         "aov": True},
        # the Cornell box configuration
        {"name": "cornell", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16, "depth": 5,
         "aov": False},
        # one full-HD frame of the single-mesh configuration (thin lens, 2048x1024 sky)
        {"name": "single_mesh_hd", "kind": "render", "scene": "single", "width": 1920, "height": 1080, "spp": 4,
         "depth": 8, "aov": True},
        # many scenes in one wavefront: 16 scenes of the batched configuration
        {"name": "batch16", "kind": "batch", "scenes": 16, "spp_scale": 1.0, "res_scale": 1.0, "depth": 8},
        # one step of inverse rendering: new texels, forward, loss gradient, adjoint
        {"name": "inverse_step", "kind": "inverse", "views": 4, "res": 256, "spp": 8, "tex": 512, "depth": 6},
        # loading one large mesh: upload, BVH, environment tables, and the first depth image
        {"name": "create_single", "kind": "create", "level": 8, "rays": 57600},
        # a batch service: scenes arrive as host descriptions, are rendered and dropped
        {"name": "create_render16", "kind": "create_batch", "scenes": 16, "spp": 4, "res": 256, "depth": 8},
        # the post-process chain and 8-bit images of a full-HD frame
        {"name": "display_hd", "kind": "post", "width": 1920, "height": 1080, "chain": "display"},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["query_host", "query_device", "render", "batch", "inverse", "create", "create_batch", "post"])
    if kind == "query_host":
        return {"kind": kind, "mesh": rng.choice(["hit", "single"]), "rays": _log(rng, 256, 129600),
                "order": rng.choice(["random", "camera"])}
    if kind == "query_device":
        return {"kind": kind, "mesh": rng.choice(["hit", "single"]), "rays": _log(rng, 4096, 2000000),
                "order": rng.choice(["random", "camera"]), "any": rng.random() < 0.5}
    if kind == "render":
        scene = rng.choice(["materials", "cornell", "single", "emitters"])
        return {"kind": kind, "scene": scene, "width": _log(rng, 48, 1024), "height": _log(rng, 48, 768),
                "spp": rng.randint(1, 9), "depth": rng.randint(3, 10), "aov": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 16), "spp_scale": rng.choice([0.25, 0.5, 1.0]),
                "res_scale": round(rng.uniform(0.3, 1.0), 3), "depth": rng.randint(4, 8)}
    if kind == "inverse":
        return {"kind": kind, "views": rng.randint(1, 4), "res": _log(rng, 48, 256), "spp": rng.randint(2, 8),
                "tex": rng.choice([64, 200, 512]), "depth": rng.randint(3, 6)}
    if kind == "create":
        return {"kind": kind, "level": rng.randint(4, 8), "rays": _log(rng, 1000, 57600)}
    if kind == "create_batch":
        return {"kind": kind, "scenes": rng.randint(2, 16), "spp": rng.randint(1, 4), "res": _log(rng, 64, 256),
                "depth": rng.randint(4, 8)}
    return {"kind": kind, "width": _log(rng, 64, 1920), "height": _log(rng, 64, 1080),
            "chain": rng.choice(["display", "tonemap"])}


# ---- what a program has in hand --------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _ctx() -> fb.Context:
    return fb.Context(0)


class _State:
    """One case's inputs; its scenes are destroyed with it."""

    def __init__(self, case, **kw):
        self.case = case
        self.scenes = []
        self.__dict__.update(kw)

    def __del__(self):
        for s in self.scenes:
            try:
                s.destroy()
            except Exception:
                pass


@functools.lru_cache(maxsize=None)
def _icosphere(level: int):
    v, f = synth.displaced_icosphere(level, 1, amp=0.05)
    return v, f


def _rotation(rng) -> np.ndarray:
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                     [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                     [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])


@functools.lru_cache(maxsize=None)
def _sky(w: int, h: int, peak: float, sigma: float) -> np.ndarray:
    return synth.sky_env(w, h, 3, sun_peak=peak, sun_sigma_deg=sigma)


@functools.lru_cache(maxsize=None)
def _single_base(level: int):
    """The single-mesh workload at one subdivision level, without its sky."""
    return synth.single_mesh_scene(level=level, env_w=8, env_h=4)


def _single_spec(level: int, rng, width=64, height=36, spp=1, depth=8, env=(2048, 1024)):
    """The single-mesh workload turned by a random rotation, with its full sky."""
    base = _single_base(level)
    m = base.objects[0]
    v = (m.vertices.astype(np.float64) @ _rotation(rng).T).astype(np.float32)
    spec = synth.SceneSpec(dict(base.camera, aspect=width / height), dict(base.renderer, width=width, height=height, spp=spp,
                                                                        depth=depth), base.materials,
                           [Mesh(v, m.faces, m.material, vattr=m.vattr)], base.lights, {"sky": _sky(*env, 5e4, 0.5)})
    return spec


def _query_spec(mesh: str, rng):
    if mesh == "single":
        spec = synth.single_mesh_hit_scene(1)
        v, f = _icosphere(8)
        spec.objects = [Mesh((v @ _rotation(rng).T).astype(np.float32), f, "m0")]
        return spec
    return synth.hit_scene(int(rng.integers(1 << 20)), level=5, spheres=6)


def _rays(spec, case, rng) -> np.ndarray:
    n = case["rays"]
    if case["order"] == "camera":
        nx = max(1, int(round(math.sqrt(n * 16.0 / 9.0))))
        ny = -(-n // nx)
        return synth.pinhole_rays(rng, spec.camera, nx, ny)[:n]
    return synth.random_rays(rng, n, (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5))


def _batch_specs(n: int, rng, depth: int, res=None, spp=None):
    base = int(rng.integers(1 << 16)) * 64
    out = []
    for i in range(n):
        out.append(synth.batch_scene(base + i, res=res(i), spp=spp(i), depth=depth))
    return out


def _batch_size(case, i):
    res = max(16, int(round((128, 256, 384, 512)[i % 4] * case["res_scale"])))
    return res, max(1, int((4, 16, 64)[i % 3] * case["spp_scale"]))


def _tuning(samples: float) -> fb.Tuning:
    """A tuning as autotune_batch returns it, kept by the program from one call to the next."""
    pool = 1 << 20
    while pool < (1 << 24) and pool * 2 <= samples:
        pool *= 2
    return fb.Tuning(pool, 256, 256, 8, 0, 0)


def _smooth(rng, res: int, lo: float, hi: float) -> np.ndarray:
    """res x res x 3 smooth random texels in [lo, hi] (16 x 16 noise, bilinearly enlarged)."""
    t = torch.from_numpy(rng.uniform(lo, hi, (1, 3, 16, 16)).astype(np.float32))
    t = torch.nn.functional.interpolate(t, size=(res, res), mode="bilinear", align_corners=True)
    return np.ascontiguousarray(t[0].permute(1, 2, 0).numpy())


def _post_inputs(case, seed: int):
    """A noisy frame with a smooth base, sharp edges and fireflies, and its guides."""
    rng = np.random.default_rng([seed, 77])
    h, w = case["height"], case["width"]
    y, x = np.meshgrid(np.linspace(0, 1, h), np.linspace(0, 1, w), indexing="ij")
    a, b = rng.uniform(2, 6, 2)
    edge = (np.sin(a * 3 * x + y) + np.cos(b * 3 * y - x) > 0.2).astype(np.float32)
    base = np.stack([0.3 + 0.4 * x, 0.5 * y + 0.2 * edge, 0.2 + 0.3 * edge], -1)
    rgb = base * rng.gamma(4.0, 0.25, (h, w, 1)) + (rng.random((h, w, 1)) < 1e-3) * 40.0
    alb = np.clip(base + 0.02 * rng.normal(size=(h, w, 3)), 0, 1)
    nrm = np.stack([np.sin(a * x), np.cos(b * y), 0.5 + edge], -1) * rng.uniform(0.9, 1.0, (h, w, 1))
    return rgb.astype(np.float32), alb.astype(np.float32), nrm.astype(np.float32)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 11])
    ctx, kind = _ctx(), case["kind"]
    if kind in ("query_host", "query_device"):
        spec = _query_spec(case["mesh"], rng)
        st = _State(case, rays=_rays(spec, case, rng))
        if kind == "query_device":
            n = case["rays"]
            if case["any"]:
                st.rays[:, 7] = rng.uniform(0.2, 2.0, n).astype(np.float32)
            st.rays = torch.from_numpy(st.rays).cuda()
            st.obj = torch.empty(n, dtype=torch.int32, device="cuda")
            st.t = torch.empty(n, dtype=torch.float32, device="cuda")
            st.occ = torch.empty(n, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
        st.scenes = [ctx.create_scene(spec.to_desc())]
        return st
    if kind == "render":
        w, h = case["width"], case["height"]
        if case["scene"] == "single":
            spec = _single_spec(8, rng, w, h, case["spp"], case["depth"])
        else:
            if case["scene"] == "materials":
                spec = synth.material_scene(int(rng.integers(1 << 20)))
            elif case["scene"] == "emitters":
                spec = synth.emitters_scene(accelerator="embree")
            else:
                spec = synth.cornell()
            spec.renderer.update(width=w, height=h, spp=case["spp"], depth=case["depth"])
            spec.camera["aspect"] = w / h
            spec.camera["pos"] = [p + float(rng.uniform(-0.05, 0.05)) for p in spec.camera["pos"]]
        st = _State(case, cam=spec.camera_struct(), params=spec.render_params(seed=int(rng.integers(1 << 40))))
        st.scenes = [ctx.create_scene(spec.to_desc())]
        return st
    if kind == "batch":
        specs = _batch_specs(case["scenes"], rng, case["depth"], lambda i: _batch_size(case, i)[0],
                             lambda i: _batch_size(case, i)[1])
        st = _State(case, cams=[s.camera_struct() for s in specs],
                    params=[s.render_params(seed=int(rng.integers(1 << 40))) for s in specs])
        st.out = [np.zeros(p.out_shape() + (3,), np.float32) for p in st.params]
        st.tuning = _tuning(sum(p.out_pixels() * p.spp for p in st.params))
        st.scenes = ctx.create_scenes([s.to_desc() for s in specs])
        return st
    if kind == "inverse":
        spec = synth.inverse_scene(tex_res=case["tex"], res=case["res"], spp=case["spp"], depth=case["depth"], target=False)
        holder = spec.to_desc()
        st = _State(case, index=holder.texture_index)
        st.base, st.rm = _smooth(rng, case["tex"], 0.1, 0.9), _smooth(rng, case["tex"], 0.1, 0.9)
        st.cams = [camera_struct(c) for c in synth.inverse_views(case["views"], int(rng.integers(1 << 20)))]
        st.params = [spec.render_params(seed=int(rng.integers(1 << 40))) for _ in st.cams]
        st.params_adj = [spec.render_params(seed=int(rng.integers(1 << 40))) for _ in st.cams]
        st.target = [_smooth(rng, case["res"], 0.2, 1.5) for _ in st.cams]
        st.out = [np.zeros(p.out_shape() + (3,), np.float32) for p in st.params]
        st.tuning = _tuning(sum(p.out_pixels() * p.spp for p in st.params))
        st.scenes = [ctx.create_scene(holder)]
        return st
    if kind == "create":
        spec = _single_spec(case["level"], rng)
        return _State(case, holder=spec.to_desc(), rays=_rays(spec, {"rays": case["rays"], "order": "camera"}, rng))
    if kind == "create_batch":
        specs = _batch_specs(case["scenes"], rng, case["depth"], lambda i: case["res"], lambda i: case["spp"])
        st = _State(case, holders=[s.to_desc() for s in specs], cams=[s.camera_struct() for s in specs],
                    params=[s.render_params(seed=int(rng.integers(1 << 40))) for s in specs])
        st.out = [np.zeros(p.out_shape() + (3,), np.float32) for p in st.params]
        st.tuning = _tuning(sum(p.out_pixels() * p.spp for p in st.params))
        return st
    rgb, alb, nrm = _post_inputs(case, seed)
    return _State(case, rgb=rgb, alb=alb, nrm=nrm)


# ---- one pass ----------------------------------------------------------------------------


def run(st):
    case, ctx = st.case, _ctx()
    kind = case["kind"]
    if kind == "query_host":
        return st.scenes[0].trace_closest(st.rays)
    if kind == "query_device":
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        h, n = st.scenes[0].h, case["rays"]
        if case["any"]:
            ctx.check(ctx.lib.fm_trace_any(ctx.h, h, p(st.rays), n, p(st.occ), fb.FM_FLAG_DEVICE_PTRS))
            return st.occ
        ctx.check(ctx.lib.fm_trace_closest(ctx.h, h, p(st.rays), n, p(st.obj), p(st.t), fb.FM_FLAG_DEVICE_PTRS))
        return st.obj, st.t
    if kind == "render":
        rgb, alb, nrm, _ = st.scenes[0].render(st.cam, st.params, want_aov=case["aov"])
        return rgb, alb, nrm
    if kind == "batch":
        return ctx.render_batch(st.scenes, st.cams, st.params, tuning=st.tuning, out=st.out)[0]
    if kind == "inverse":
        sc = st.scenes[0]
        sc.update_texture(st.index["basecolor"], st.base)
        sc.update_texture(st.index["rm"], st.rm)
        img = ctx.render_batch([sc] * len(st.cams), st.cams, st.params, tuning=st.tuning, out=st.out)[0]
        scale = np.float32(2.0 / sum(a.size for a in img))
        d = [(a - t) * scale for a, t in zip(img, st.target)]
        shape = st.base.shape[:2]
        grads = sc.render_adjoint(st.cams, st.params_adj, d, {st.index["basecolor"]: shape, st.index["rm"]: shape})[0]
        return img, [grads[st.index["basecolor"]], grads[st.index["rm"]]]
    if kind == "create":
        sc = ctx.create_scene(st.holder)
        out = sc.trace_closest(st.rays)
        sc.destroy()
        return out
    if kind == "create_batch":
        scenes = ctx.create_scenes(st.holders)
        img = ctx.render_batch(scenes, st.cams, st.params, tuning=st.tuning, out=st.out)[0]
        for s in scenes:
            s.destroy()
        return img
    return ctx.postprocess(CHAINS[case["chain"]], st.rgb, st.alb, st.nrm)


# ---- what a pass cannot do without ---------------------------------------------------------

_NODE, _PRIM, _VERTEX = 8 * 16.0, 60.0, 400.0   # operations: one 8-wide node, one triangle test, shading one vertex
_TRI_BYTES = 36.0


def _ray_ops(tris: float) -> float:
    return math.ceil(math.log(max(tris, 8) / 4.0, 8)) * _NODE + 2 * _PRIM


def _path_ops(tris: float, depth: int, lights: int) -> float:
    """One camera path: about half of `depth` vertices (roulette, escapes), each with a
    continuation ray, an MIS ray and a shadow ray per light."""
    v = 0.5 * depth
    return v * ((2 + lights) * _ray_ops(tris) + _VERTEX)


def work(case):
    kind = case["kind"]
    single = 20.0 * 4 ** 8
    if kind in ("query_host", "query_device"):
        tris = single if case["mesh"] == "single" else 20.0 * 4 ** 5
        n = case["rays"]
        return {"bytes": 32.0 * n + (1.0 if case.get("any") else 8.0) * n, "flops": n * _ray_ops(tris)}
    if kind == "render":
        tris = {"single": single, "materials": 1280.0, "cornell": 12.0, "emitters": 500.0}[case["scene"]]
        px = case["width"] * case["height"]
        return {"bytes": px * 12.0 * (3 if case["aov"] else 1) + tris * _TRI_BYTES,
                "flops": px * case["spp"] * _path_ops(tris, case["depth"], {"single": 1, "materials": 3}.get(case["scene"], 1))}
    if kind in ("batch", "create_batch"):
        tris, b, f = 2.0e4, 0.0, 0.0
        for i in range(case["scenes"]):
            res, spp = _batch_size(case, i) if kind == "batch" else (case["res"], case["spp"])
            b += res * res * 12.0 + tris * _TRI_BYTES
            f += res * res * spp * _path_ops(tris, case["depth"], 2)
            if kind == "create_batch":
                f += tris * 20 * 24.0
                b += 512 * 256 * 12.0
        return {"bytes": b, "flops": f}
    if kind == "inverse":
        px, tex = case["views"] * case["res"] ** 2, case["tex"] ** 2
        return {"bytes": px * 12.0 * 3 + tex * 2 * (12.0 + 24.0) + 119600 * _TRI_BYTES,
                "flops": px * case["spp"] * 3 * _path_ops(119600.0, case["depth"], 2)}
    if kind == "create":
        tris = 20.0 * 4 ** case["level"]
        # uploaded triangles, attributes and sky; a binned sweep per level of the tree
        return {"bytes": tris * (36.0 + 72.0 + 16.0) + 2048 * 1024 * 12.0 + case["rays"] * 40.0,
                "flops": tris * math.log2(tris) * 24.0 + case["rays"] * _ray_ops(tris)}
    px = case["width"] * case["height"]
    denoise = case["chain"] == "display"
    return {"bytes": px * (24.0 + 24.0 + 9.0), "flops": px * ((5 * 25 * 40.0 if denoise else 0.0) + 60.0)}


# ---- the same in 64 bits ---------------------------------------------------------------------


def _exact_hits(spec, rays):
    """Closest hits by testing every primitive (Moeller-Trumbore, sphere quadratic), float64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h = spec.to_desc()
    tri = [h.tri_pos.reshape(-1, 3, 3)]
    for r in h.rect_pts.reshape(-1, 4, 3):
        tri.append(r[[0, 1, 2]][None])
        tri.append(r[[2, 3, 0]][None])
    tri = torch.from_numpy(np.concatenate(tri)).to(dev, torch.float64)
    obj = torch.from_numpy(np.concatenate([h.tri_object, np.repeat(h.rect_object, 2)])).to(dev)
    r = torch.from_numpy(rays).to(dev, torch.float64)
    o, d = r[:, None, 0:3], r[:, None, 4:7]
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device=dev)
    which = torch.full((len(rays),), -1, dtype=torch.int32, device=dev)
    step = max(1, (1 << 22) // len(rays))
    for i in range(0, len(tri), step):
        v0, e1, e2 = tri[None, i:i + step, 0], tri[None, i:i + step, 1], tri[None, i:i + step, 2]
        e1, e2 = e1 - v0, e2 - v0
        p = torch.linalg.cross(d.expand(-1, e2.shape[1], -1), e2.expand(len(rays), -1, -1))
        det = (e1 * p).sum(-1)
        s = o - v0
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1.expand(len(rays), -1, -1))
        v = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0), t, math.inf)
        m, k = t.min(1)
        which = torch.where(m < best, obj[i + k].to(torch.int32), which)
        best = torch.minimum(best, m)
    for rad, x, ob in zip(h.sphere_radius, h.sphere_xform.reshape(-1, 4, 4), h.sphere_object):
        oc = r[:, 0:3] - torch.from_numpy(x[:3, 3]).to(dev, torch.float64)
        dd = r[:, 4:7]
        a, b, c = (dd * dd).sum(-1), 2 * (dd * oc).sum(-1), (oc * oc).sum(-1) - float(rad) ** 2
        disc = torch.sqrt(b * b - 4 * a * c)
        t0, t1 = (-b - disc) / (2 * a), (-b + disc) / (2 * a)
        t = torch.where(t0 >= 0, t0, torch.where(t1 >= 0, t1, math.inf))
        t = torch.where(torch.isnan(t), math.inf, t)
        which = torch.where(t < best, torch.full_like(which, int(ob)), which)
        best = torch.minimum(best, t)
    return which.cpu().numpy(), best.cpu().numpy()


def _exact_post(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rgb, alb, nrm = (torch.from_numpy(a).to(dev, torch.float64) for a in _post_inputs(case, seed))
    h, w, _ = rgb.shape
    for kind, lum in CHAINS[case["chain"]]:
        if kind == fb.FM_POST_DENOISE:
            n = nrm / torch.where(nrm.norm(dim=-1, keepdim=True) > 0, nrm.norm(dim=-1, keepdim=True), torch.ones_like(nrm[..., :1]))
            k5 = [1 / 16, 4 / 16, 6 / 16, 4 / 16, 1 / 16]
            for level in range(5):
                step, sc = 1 << level, 0.5 / (1 << level)
                t = rgb / (1 + rgb.clamp(min=0))
                acc, ws = torch.zeros_like(rgb), torch.zeros_like(rgb[..., :1])
                for dy in range(-2, 3):
                    for dx in range(-2, 3):
                        y0, y1 = max(0, -dy * step), min(h, h - dy * step)
                        x0, x1 = max(0, -dx * step), min(w, w - dx * step)
                        if y0 >= y1 or x0 >= x1:
                            continue
                        a = (slice(y0, y1), slice(x0, x1))
                        b = (slice(y0 + dy * step, y1 + dy * step), slice(x0 + dx * step, x1 + dx * step))
                        wt = torch.exp(-((t[b] - t[a]) ** 2).sum(-1) / sc ** 2
                                       - (1 - (n[a] * n[b]).sum(-1)).clamp(min=0) / 0.35 ** 2
                                       - ((alb[b] - alb[a]) ** 2).sum(-1) / 0.1 ** 2)[..., None] * (k5[dx + 2] * k5[dy + 2])
                        acc[a] += rgb[b] * wt
                        ws[a] += wt
                rgb = acc / ws
        elif kind == fb.FM_POST_TONEMAP:
            core = lambda x: (x * (0.22 * x + 0.10 * 0.30) + 0.20 * 0.01) / (x * (0.22 * x + 0.30) + 0.20 * 0.30) - 0.01 / 0.30  # noqa: E731
            rgb = core(1.6 * rgb * float(np.float32(lum))) / core(11.2)
        else:
            rgb = torch.where(rgb <= 0.0031308, 12.92 * rgb, 1.055 * rgb.clamp(min=0) ** (1 / 2.4) - 0.055)
    return rgb.cpu().numpy(), None, None, None


def exact(case, seed):
    if case["kind"] == "post":
        return _exact_post(case, seed)
    if case["kind"] == "query_host" and case["mesh"] == "hit" and case["rays"] <= 20000:
        rng = np.random.default_rng([seed, 11])
        spec = _query_spec(case["mesh"], rng)
        return _exact_hits(spec, _rays(spec, case, rng))
    # Monte-Carlo images have no value of their own per seed; the large meshes have no search without a tree
    return None
