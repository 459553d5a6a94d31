"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the public entry points of ``cadise_gb300`` (the ctypes view of
``include/cadise_gpu.h``): ray queries on host and device buffers, frames of one scene, a batch of
uneven scenes, the allocation-free preview frame, the whole one-shot flow of the command line, and
the differentiable-rendering iteration.  Scenes come from ``cadise_gb300.scenes``; sizes are those of
the repository's configurations, tests and benchmark, or smaller and odd ones of the same kinds.

A case's ``tuned`` says whether the program sets the tuning that ``bench.py`` reports for the
million-triangle frame (what a program does that has run ``cgpu_autotune`` once), or takes a new
context as it is (the command line, INTEGRATION.md's examples).
"""
import math

import numpy as np
import torch

import cadise_gb300 as cg
from cadise_gb300 import abi, scenes

RAY_EPS = 1e-3
FLT_MAX = 3.402823466e38

# cgpu_autotune's choice for the 1920 x 1080 million-triangle frame, as bench.py prints it
BENCH_TUNING = {"block_trace": 64, "block_shade": 128, "max_paths": 1 << 24, "traversal": 3, "reorder": 0,
                "refill_closest": 28, "refill_any": 32}


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # A picking tool or a baker that asks for a handful of rays at a time: host buffers both ways.
        {"name": "closest_host_257", "kind": "closest_host", "spheres": 10, "sub": 2, "rays": 257},
        # Baking / visibility jobs over resident buffers: incoherent rays through the million-triangle field.
        {"name": "closest_dev_field1m", "kind": "closest_device", "spheres": 200, "sub": 4, "rays": 3_000_001},
        # The same for visibility alone, with rays that end at a second point.
        {"name": "any_dev_field1m", "kind": "any_device", "spheres": 200, "sub": 4, "rays": 2_000_003},
        # The first configuration: Cornell box, 256 x 256, 16 spp, depth 6, as the command line renders it.
        {"name": "cornell_256_16spp", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 6, "tuned": False},
        # The shipped kind of scene (analytic spheres, plastic, Phong, mirrors, glass; Gaussian film filter)
        # on an odd frame.
        {"name": "spheres_filtered_333", "kind": "render", "scene": "spheres", "width": 333, "height": 251, "spp": 9,
         "depth": 8, "tuned": False},
        # A preview inside a loop that may not allocate: one small frame, few samples.
        {"name": "noalloc_preview", "kind": "noalloc", "width": 320, "height": 181, "spp": 2, "depth": 8},
        # The headline frame: 1,024,018 triangles, 1920 x 1080, depth 12 with roulette; 16 of its 64 spp a pass.
        {"name": "field1m_1080p", "kind": "render", "scene": "field", "spheres": 200, "sub": 4, "width": 1920,
         "height": 1080, "spp": 16, "depth": 12, "tuned": True},
        # The stress configuration's kind: HDR sky, 64 lights, GGX palette, depth 32, 2 M triangles.
        {"name": "env2m_1080p", "kind": "render", "scene": "env", "spheres": 400, "sub": 4, "width": 1920,
         "height": 1080, "spp": 4, "depth": 32, "tuned": True},
        # Uneven scenes in one call, each with its own size, sample count and depth.
        {"name": "batch_12_scenes", "kind": "batch", "count": 12, "sizes": 3, "tri_lo": 10_000, "tri_hi": 200_000,
         "tuned": True},
        # One differentiable-rendering iteration of the fourth configuration: parameters in, 512 x 512 x 32 spp
        # forward, L2 loss, path-replay adjoint, gradients out.
        {"name": "adjoint_512_32spp", "kind": "adjoint", "spheres": 20, "sub": 4, "tex": 256, "width": 512,
         "height": 512, "spp": 32, "depth": 6, "tuned": True},
        # The same loop on a small problem, where each iteration is short.
        {"name": "adjoint_small", "kind": "adjoint", "spheres": 12, "sub": 2, "tex": 33, "width": 127, "height": 95,
         "spp": 8, "depth": 4, "tuned": False},
        # What the command line does for every scene file: upload (BVH build), render, read the film, release.
        {"name": "oneshot_102k", "kind": "oneshot", "spheres": 20, "sub": 4, "width": 640, "height": 360, "spp": 4,
         "depth": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest_host", "closest_device", "any_device", "render", "render", "render", "noalloc",
                       "batch", "adjoint", "adjoint", "oneshot"])
    if kind == "closest_host":
        return {"kind": kind, "spheres": rng.randint(3, 12), "sub": 2, "rays": _log(rng, 1, 600)}
    if kind in ("closest_device", "any_device"):
        return {"kind": kind, "spheres": _log(rng, 5, 200), "sub": rng.choice([3, 4]),
                "rays": _log(rng, 1000, 3_000_000)}
    if kind == "noalloc":
        return {"kind": kind, "width": _log(rng, 40, 480), "height": _log(rng, 40, 480), "spp": _log(rng, 1, 12),
                "depth": rng.randint(3, 12)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 12), "sizes": rng.randint(1, 1 << 20), "tri_lo": 10_000,
                "tri_hi": _log(rng, 20_000, 200_000), "tuned": rng.random() < 0.5}
    if kind == "adjoint":
        return {"kind": kind, "spheres": _log(rng, 9, 20), "sub": rng.choice([2, 3, 4]), "tex": _log(rng, 16, 256),
                "width": _log(rng, 64, 512), "height": _log(rng, 64, 512), "spp": _log(rng, 2, 32),
                "depth": rng.randint(2, 6), "tuned": rng.random() < 0.5}
    if kind == "oneshot":
        return {"kind": kind, "spheres": _log(rng, 2, 20), "sub": 4, "width": _log(rng, 64, 640),
                "height": _log(rng, 64, 360), "spp": rng.randint(1, 4), "depth": rng.randint(3, 8)}
    scene = rng.choice(["cornell", "spheres", "field", "field", "env"])
    c = {"kind": "render", "scene": scene}
    if scene in ("field", "env"):
        c.update(spheres=_log(rng, 8, 200), sub=rng.choice([3, 4]))
    c.update(width=_log(rng, 96, 1920), height=_log(rng, 64, 1080), spp=_log(rng, 1, 16),
             depth=rng.choice([4, 6, 8, 12, 16]), tuned=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ scenes --
def _field(case, seed, **kw):
    n = case["spheres"]
    return scenes.icosphere_field(n_spheres=n, subdivision=case["sub"], seed=seed,
                                  box=100.0 * (n / 200.0) ** (1 / 3), **kw)


def _frame(case):
    return {"width": case["width"], "height": case["height"], "spp": case["spp"], "max_depth": case["depth"]}


def _scene(case, seed):
    kind = case.get("scene")
    if kind == "cornell":
        return scenes.cornell_box(**_frame(case))
    if kind == "spheres":
        s = scenes.sphere_box(**_frame(case))
        s.film_filter = scenes.FilmFilter(type="gaussian", width=4.0, height=4.0, sigma_x=0.5, sigma_y=0.5)
        return s
    if kind == "env":
        return scenes.env_field(n_spheres=case["spheres"], subdivision=case["sub"], seed=seed, sky=(1024, 512),
                                **_frame(case))
    return _field(case, seed, **_frame(case))


def _batch_sizes(case):
    """Spheres, subdivision and frame of each scene of a batch, as scenes.batch_scenes spreads them, at half
    its resolution (and three rows less) and an eighth of its samples."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        tris = math.exp(rng.uniform(math.log(case["tri_lo"]), math.log(case["tri_hi"])))
        sub = 4 if tris >= 51_200 else 3
        res = int(rng.choice([128, 256, 512, 1024])) // 2
        out.append({"spheres": max(1, int(round(tris / (20 * 4 ** sub)))), "sub": sub, "width": res, "height": res - 3,
                    "spp": max(1, int(rng.choice([4, 16, 64, 256])) // 8), "depth": int(rng.choice([4, 8, 16]))})
    return out


def _context(case):
    stream = torch.cuda.Stream()
    ctx = cg.Context(device=0, stream=stream.cuda_stream)
    if case.get("tuned"):
        ctx.set_tuning_dict(BENCH_TUNING)
    return {"kind": case["kind"], "case": case, "stream": stream, "ctx": ctx}


def _host_rays(case, seed, bounds):
    """Incoherent rays: origins in the scene's box, directions over the sphere."""
    rng = np.random.default_rng([seed, 77])
    lo, hi = bounds
    n = case["rays"]
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = lo + (hi - lo) * rng.random((n, 3))
    rays[:, 3] = RAY_EPS
    d = rng.standard_normal((n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = FLT_MAX
    return rays


def _query_box(case):
    """The cube of the spheres' centres (the ground plane reaches further)."""
    box = 100.0 * (case["spheres"] / 200.0) ** (1 / 3)
    return np.zeros(3), np.full(3, box)


def _device_rays(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    lo, hi = (torch.tensor(v, dtype=torch.float32, device="cuda") for v in _query_box(case))
    n = case["rays"]
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    org = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    if case["kind"] == "any_device":  # visibility between two points of the scene
        d = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda") - org
        dist = d.norm(dim=1)
        rays[:, 7] = dist - RAY_EPS
        rays[:, 4:7] = d / dist.clamp_min(1e-6)[:, None]
    else:
        d = torch.randn((n, 3), generator=g, device="cuda")
        rays[:, 4:7] = d / d.norm(dim=1).clamp_min(1e-6)[:, None]
        rays[:, 7] = FLT_MAX
    rays[:, 0:3] = org
    rays[:, 3] = RAY_EPS
    return rays


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    st = _context(case)
    ctx, kind = st["ctx"], case["kind"]
    st["seed"] = seed
    if kind in ("closest_host", "closest_device", "any_device"):
        st["sid"] = ctx.upload(_field(case, seed, width=64, height=64, spp=1, max_depth=1))
        if kind == "closest_host":
            st["rays"] = _host_rays(case, seed, _query_box(case))
        else:
            st["rays"] = _device_rays(case, seed)
            n = case["rays"]
            st["out"] = (torch.zeros((n, 4), dtype=torch.int32, device="cuda") if kind == "closest_device"
                         else torch.zeros(n, dtype=torch.uint8, device="cuda"))
    elif kind == "render":
        st["sid"] = ctx.upload(_scene(case, seed))
        npix = case["width"] * case["height"]
        film = torch.zeros(npix * 7, dtype=torch.float64, pin_memory=True)  # read back as bench.py does
        st["film"] = film
        st["arrays"] = [film.numpy()[a * npix:b * npix] for a, b in ((0, 3), (3, 6), (6, 7))]
    elif kind == "noalloc":
        st["sid"] = ctx.upload(scenes.power_field(seed=seed, **_frame(case)))
    elif kind == "batch":
        sizes = _batch_sizes(case)
        st["sids"] = [ctx.upload(_field(c, 1000 * seed + i, **_frame(c))) for i, c in enumerate(sizes)]
        st["counts"] = [c["spp"] for c in sizes]
    elif kind == "adjoint":
        spec = scenes.diff_scene(n_spheres=case["spheres"], subdivision=case["sub"], tex_size=case["tex"], seed=seed,
                                 n_conductors=min(8, case["spheres"] - 1), **_frame(case))
        sid = st["sid"] = ctx.upload(spec)
        tex, rough, rad = st["params"] = ctx.get_params(sid)
        # target from perturbed parameters (albedo +-0.2, roughness +-0.15)
        rng = np.random.default_rng(seed)
        ctx.set_params(sid, np.clip(tex + rng.uniform(-0.2, 0.2, tex.shape), 0.02, 0.98).astype(np.float32),
                       np.clip(rough + rng.uniform(-0.15, 0.15, rough.shape), 0.05, 1.0).astype(np.float32), rad)
        st["target"] = ctx.adjoint_forward(sid, 4 * case["spp"], seed + 77)
        st["grad_img"] = np.empty_like(st["target"])
    else:
        st["flat"] = abi.flatten(_field(case, seed, **_frame(case)))
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- run --
def run(st):
    ctx, kind, case = st["ctx"], st["kind"], st["case"]
    if kind == "closest_host":
        prim, t, u, v = ctx.trace_closest(st["sid"], st["rays"])
        return {"prim": prim, "t": t, "u": u, "v": v}
    if kind == "closest_device":
        out = st["out"]
        ctx._check(ctx.L.cgpu_trace_closest_device(ctx.h, st["sid"], st["rays"].data_ptr(), case["rays"],
                                                   out.data_ptr()))
        f = out.view(torch.float32)
        return {"prim": out[:, 1], "t": f[:, 0], "u": f[:, 2], "v": f[:, 3]}
    if kind == "any_device":
        ctx._check(ctx.L.cgpu_trace_any_device(ctx.h, st["sid"], st["rays"].data_ptr(), case["rays"],
                                               st["out"].data_ptr()))
        return {"occluded": st["out"]}
    if kind == "render":
        sid = st["sid"]
        ctx.film_clear(sid)
        ctx.render([sid], 0, case["spp"], seed=st["seed"], sync=False)
        ctx.film_read_into(sid, *st["arrays"])
        s, q, n = st["arrays"]
        return {"sum": s, "sum_sq": q, "count": n}
    if kind == "noalloc":
        sid = st["sid"]
        ctx.film_clear(sid)
        ctx.render_noalloc(sid, 0, case["spp"], seed=st["seed"], sync=False)
        s, q, n = ctx.film_read(sid)
        return {"sum": s, "sum_sq": q, "count": n}
    if kind == "batch":
        for sid in st["sids"]:
            ctx.film_clear(sid)
        ctx.render(st["sids"], 0, st["counts"], seed=st["seed"], sync=False)
        films = [ctx.film_read(sid) for sid in st["sids"]]
        return {"sum": [f[0] for f in films], "sum_sq": [f[1] for f in films], "count": [f[2] for f in films]}
    if kind == "adjoint":
        sid, spp, seed = st["sid"], case["spp"], st["seed"]
        ctx.set_params(sid, *st["params"])
        img = ctx.adjoint_forward(sid, spp, seed)
        g = st["grad_img"]
        np.subtract(img, st["target"], out=g)
        g *= np.float32(2.0 / g.size)
        gt, gr, gl = ctx.adjoint_backward(sid, spp, seed, g)
        return {"image": img, "texels": gt, "roughness": gr, "radiance": gl}
    sid = ctx.upload(st["flat"])
    ctx.render([sid], 0, case["spp"], seed=st["seed"], sync=False)
    s, q, n = ctx.film_read(sid)
    ctx.release(sid)
    return {"sum": s, "sum_sq": q, "count": n}


# -------------------------------------------------------------------- work --
def _ray_flops(tris):
    """Arithmetic that one ray cannot do without: a 4-wide tree's levels, four boxes of 6 multiply-adds
    each, and two triangle tests."""
    return max(1.0, math.log(max(tris, 4), 4)) * 4 * 12 + 2 * 45


def _path_flops(depth, tris):
    """Rays of one path sample: the primary ray, and at each further vertex (half the paths end at each)
    a continuation and a light ray, with some 200 operations of shading a vertex."""
    vertices = sum(0.5 ** k for k in range(min(depth, 12)))
    return 2 * vertices * _ray_flops(tris) + 200 * vertices


def work(case):
    kind = case["kind"]
    if kind == "batch":
        each = [work(dict(c, kind="render", scene="field")) for c in _batch_sizes(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    scene = case.get("scene", "field")
    tris = {"cornell": 36, "spheres": 30}.get(scene, case.get("spheres", 10) * 20 * 4 ** case.get("sub", 2))
    if "rays" in case:
        out = 1 if kind == "any_device" else 16
        return {"bytes": 36.0 * tris + (32 + out) * case["rays"], "flops": case["rays"] * _ray_flops(tris)}
    npix, spp, depth = case["width"] * case["height"], case["spp"], case["depth"]
    if kind == "adjoint":
        params = 3 * case["tex"] ** 2
        return {"bytes": 36.0 * tris + 24 * npix + 12 * params, "flops": 2 * npix * spp * _path_flops(depth, tris)}
    return {"bytes": 36.0 * tris + 56 * npix, "flops": npix * spp * _path_flops(depth, tris)}


# ------------------------------------------------------------------- exact --
def _exact_closest(case, seed):
    """Closest hits by brute force in 64 bits over every primitive of the scene."""
    spec = _field(case, seed, width=64, height=64, spp=1, max_depth=1)
    rays = _host_rays(case, seed, _query_box(case)).astype(np.float64)
    o, d = rays[:, :3], rays[:, 4:7]
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    n = len(rays)
    best, bu, bv = np.full(n, np.inf), np.zeros(n), np.zeros(n)

    def keep(ok, t, u, v):
        t = np.where(ok & (t >= RAY_EPS), t, np.inf)
        k = t.argmin(1)
        r = np.arange(n)
        near = t[r, k] < best
        best[near], bu[near], bv[near] = t[r, k][near], u[r, k][near], v[r, k][near]

    for p in spec.primitives:
        if isinstance(p, scenes.Rectangle):
            v1, vb, v3 = (np.asarray(np.float32(x), np.float64) for x in (p.v1, p.v2, p.v3))
            ea, eb = v1 - vb, v3 - vb
            nrm = np.cross(ea, eb)
            with np.errstate(divide="ignore", invalid="ignore"):
                t = ((vb - o) @ nrm / (d @ nrm))[:, None]
                q = o + d * t - vb
                la, lb = np.linalg.norm(ea), np.linalg.norm(eb)
                a, b = (q @ ea / la)[:, None], (q @ eb / lb)[:, None]
            keep((a >= 0) & (a <= la) & (b >= 0) & (b <= lb), t, a / la, b / la)  # both over |eA|
        else:
            v = p.positions.reshape(-1, 3, 3).astype(np.float64)
            a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
            pv = np.cross(d[:, None], e2[None])
            with np.errstate(divide="ignore", invalid="ignore"):
                inv = 1.0 / (pv * e1[None]).sum(2)
                tv = o[:, None] - a[None]
                u = (pv * tv).sum(2) * inv
                qv = np.cross(tv, e1[None])
                w = (qv * d[:, None]).sum(2) * inv
                t = (qv * e2[None]).sum(2) * inv
            keep((u >= 0) & (w >= 0) & (u + w <= 1), t, u, w)
    miss = np.isinf(best)
    best[miss] = 0.0
    return {"prim": None, "t": best, "u": bu, "v": bv}


def exact(case, seed):
    """Closest hits of the host queries; of a frame, what its Monte Carlo sums leave determined: with the
    box filter every pixel counts every sample."""
    kind = case["kind"]
    if kind == "closest_host":
        return _exact_closest(case, seed)
    if kind == "batch":
        sizes = _batch_sizes(case)
        none = [None] * len(sizes)
        return {"sum": none, "sum_sq": none,
                "count": [np.full((c["height"], c["width"]), float(c["spp"])) for c in sizes]}
    if kind in ("noalloc", "oneshot") or (kind == "render" and case["scene"] != "spheres"):
        shape = (case["height"], case["width"]) if kind != "render" else (case["height"] * case["width"],)
        return {"sum": None, "sum_sq": None, "count": np.full(shape, float(case["spp"]))}
    return None
