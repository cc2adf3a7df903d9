"""The work that a program using this framework has it do, one case per entry point and size.

Ray queries (closest and any hit, device and host buffers), the three renderers that carry a
scene script (path tracing, direct lighting, guided), batched rendering, the photon pass (map
rebuild, k nearest photons, radiance estimate) and the guide network (inference and one training
step). Scenes are the seeded procedural ones of liar_b200.scenes*; a case's seed makes the rays,
photons, network inputs or the renderer's samples. Device work runs on torch's current stream.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from liar_b200 import batch, guiding, photons, render, scenes, scenes_batch, scenes_guiding, scenes_render, tracers
from liar_b200.trace import Context, Mesh

# triangles of the displaced icosphere at each subdivision level: 20 * 4^level
LEVELS = (3, 8)
PAIRS = 3e10  # ray-triangle or query-photon pairs that the 64-bit brute force takes on


def listed():
    return [
        # the traversal workload of the benchmark: incoherent rays, as the bounces of a path tracer send
        {"name": "closest_1310k_16m", "kind": "trace", "level": 8, "rays": 16777216, "any_hit": False, "tmax": 0.0},
        # occlusion queries (shadow rays of bounded length) against a mid-sized model, an odd count
        {"name": "any_328k_2m", "kind": "trace", "level": 7, "rays": 2000003, "any_hit": True, "tmax": 0.5},
        # picking and probing: a handful of rays, where the launches count
        {"name": "closest_5k_1000", "kind": "trace", "level": 4, "rays": 1000, "any_hit": False, "tmax": 0.0},
        # a host program tracing an image's camera rays from numpy arrays
        {"name": "intersect_82k_camera", "kind": "intersect", "level": 6, "width": 641, "height": 479},
        # the plain spectral path tracer on the Cornell box, the benchmark's frame
        {"name": "path_cornell_256_16spp", "kind": "path", "width": 256, "height": 256, "spp": 16},
        # DirectLighting, the tracer of the example scripts, at an uneven resolution
        {"name": "direct_cornell_321x243_4spp", "kind": "direct", "width": 321, "height": 243, "spp": 4},
        # guided rendering with a network at hand, in the closed room lit through a slit
        {"name": "guided_slit_512_4spp", "kind": "guided", "triangles": 200000, "side": 512, "spp": 4},
        # many scenes of uneven size in one launch, four hero wavelengths
        {"name": "batch_10_scenes", "kind": "batch", "scenes": 10, "set": 0, "triangles": 200000, "side": 512, "spp": 16},
        # a photon-mapping pass at the size of a full frame: photons on surfaces, 64 nearest
        {"name": "photons_4m_1m_k64", "kind": "photons", "photons": 4000000, "queries": 1000003, "k": 64, "surface": True},
        # a small progressive pass through a volume of photons, few neighbours
        {"name": "photons_100k_20k_k16", "kind": "photons", "photons": 100000, "queries": 20001, "k": 16, "surface": False},
        # the guide network over a wave of path vertices
        {"name": "guide_eval_1m", "kind": "guide_eval", "rows": 1000000},
        # one optimiser step of the guide network with its gradient
        {"name": "guide_train_65536", "kind": "guide_train", "rows": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "intersect", "path", "direct", "guided", "batch", "photons", "photons",
                       "guide_eval", "guide_train"])
    if kind == "trace":
        any_hit = rng.random() < 0.5
        return {"kind": kind, "level": rng.randint(*LEVELS), "rays": _log(rng, 500, 16000000), "any_hit": any_hit,
                "tmax": rng.choice([0.25, 0.5, 2.0]) if any_hit else 0.0}
    if kind == "intersect":
        w = _log(rng, 64, 1920)
        return {"kind": kind, "level": rng.randint(3, 7), "width": w, "height": max(16, int(w * rng.uniform(0.5, 1.0)))}
    if kind in ("path", "direct"):
        w = _log(rng, 48, 640)
        return {"kind": kind, "width": w, "height": max(16, int(w * rng.uniform(0.5, 1.0))), "spp": rng.choice([1, 4, 9, 16])}
    if kind == "guided":
        return {"kind": kind, "triangles": _log(rng, 20000, 200000), "side": _log(rng, 64, 512), "spp": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 10), "set": rng.randint(1, 1000), "triangles": _log(rng, 20000, 200000),
                "side": _log(rng, 128, 512), "spp": _log(rng, 4, 16)}
    if kind == "photons":
        return {"kind": kind, "photons": _log(rng, 20000, 4000000), "queries": _log(rng, 2000, 1000000),
                "k": rng.choice([8, 16, 32, 50, 64]), "surface": rng.random() < 0.6}
    if kind == "guide_eval":
        return {"kind": kind, "rows": _log(rng, 300, 1000000)}
    return {"kind": kind, "rows": _log(rng, 1000, 65536)}


# ---- what a program sets up once: the context, models and flattened scenes


@functools.lru_cache(maxsize=None)
def _ctx():
    return Context(torch.cuda.current_device())


def _stream():
    return torch.cuda.current_stream().cuda_stream or guiding.CUDA_STREAM_LEGACY


@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return scenes.displaced_icosphere(levels=level, seed=0)


@functools.lru_cache(maxsize=4)
def _flat(kind, *args):
    if kind == "cornell":
        scene, cam = scenes_render.cornell_box()
        return render.flatten(scene), cam
    if kind == "slit":
        scene, cam = scenes_guiding.slit_room(*args)
        return render.flatten(scene), cam
    count, which, tris, side, spp = args
    work = scenes_batch.batch_workload(count, seed=which, tris=(10000, tris), side=(64, side), spp=(2, spp))
    return [(render.flatten(w.scene), w) for w in work]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _unit(n, g):
    """n directions uniform on the sphere."""
    u = torch.rand((n, 2), generator=g, device="cuda")
    z = 1 - 2 * u[:, 0]
    r = (1 - z * z).clamp(min=0).sqrt()
    phi = 2 * math.pi * u[:, 1]
    return torch.stack([r * phi.cos(), r * phi.sin(), z], 1)


def _random_rays(case, seed):
    """Origins uniform in 1.5 times the model's box, directions uniform on the sphere."""
    g = _gen(seed)
    v, _ = _icosphere(case["level"])
    lo, hi = torch.from_numpy(v.min(0)).cuda(), torch.from_numpy(v.max(0)).cuda()
    n = case["rays"]
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3] = (lo + hi) / 2 + 0.75 * (hi - lo) * (2 * torch.rand((n, 3), generator=g, device="cuda") - 1)
    rays[:, 3] = 0.0
    rays[:, 4:7] = _unit(n, g)
    rays[:, 7] = case["tmax"] or math.inf
    return rays


def _camera_rays(case, seed):
    """One jittered ray per pixel of a pinhole camera that looks at the model, as a numpy array."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    ys, xs = np.mgrid[0:h, 0:w]
    sx = ((xs + rng.random((h, w))) / w - 0.5).ravel()
    sy = ((ys + rng.random((h, w))) / h - 0.5).ravel() * h / w
    d = np.stack([sx, -sy, np.ones(w * h)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((w * h, 8), np.float32)
    rays[:, 0:3] = (0.1, 0.05, -2.6)
    rays[:, 4:7] = d
    rays[:, 7] = np.inf
    return rays


def _photon_inputs(case, seed):
    """Photons on a ground square (a caustic spot among even light) and a wall, or through a box;
    camera-ordered query points among them. The search radius is a few times the mean distance of
    the k-th neighbour, as an automatic radius gives it."""
    g = _gen(seed)
    n, nq, k = case["photons"], case["queries"], case["k"]

    def points(m, order):
        u = torch.rand((m, 3), generator=g, device="cuda")
        if order:  # scanlines of an image
            side = max(1, int(math.sqrt(m)))
            i = torch.arange(m, device="cuda")
            u[:, 0] = ((i % side) + u[:, 0]) / side
            u[:, 2] = ((i // side) + u[:, 2]) / ((m + side - 1) // side)
        p = u * torch.tensor([6.0, 6.0, 6.0], device="cuda") - torch.tensor([3.0, 0.0, 3.0], device="cuda")
        if case["surface"]:
            part = torch.rand(m, generator=g, device="cuda")
            wall = part < 0.2
            p[:, 1] = torch.where(wall, p[:, 1] * 0.5, 0.0)
            p[:, 2] = torch.where(wall, 3.0, p[:, 2])
            if not order:
                spot = part > 0.75
                s = 0.25 * torch.randn((m, 2), generator=g, device="cuda")
                p[:, 0] = torch.where(spot, (s[:, 0] - 0.4).clamp(-3, 3), p[:, 0])
                p[:, 2] = torch.where(spot, (s[:, 1] + 0.2).clamp(-3, 3), p[:, 2])
        return p.contiguous()

    pos, q = points(n, False), points(nq, True)
    power = torch.rand((n, 3), generator=g, device="cuda") + 0.05
    omega, normals = _unit(n, g), _unit(nq, g)
    r = 4 * math.sqrt(k * 36 / (math.pi * n)) if case["surface"] else 1.6 * (k * 216 / (4.19 * n)) ** (1 / 3)
    return pos, power, omega, q, normals, r


def _guide_inputs(rows, seed, records):
    g = _gen(seed)
    pos = torch.rand((rows, 3), generator=g, device="cuda") * 10 - 5
    parts = [pos, _unit(rows, g), _unit(rows, g)]
    if records:
        parts += [_unit(rows, g), torch.randn((rows, 1), generator=g, device="cuda").exp()]
    return torch.cat(parts, 1).contiguous()


def _weights(seed):
    """The guide's weights (f32, concatenated row-major), He-uniform with the padding rows and columns zero."""
    g = torch.Generator().manual_seed(int(seed) + 1)
    parts = []
    for rows, cols, used_rows, used_cols in ((256, 64, 225, 64),) + 4 * ((64, 64, 64, 64),) + ((64, 48, 64, 40),):
        w = torch.zeros((rows, cols))
        w[:used_rows, :used_cols] = (2 * torch.rand((used_rows, used_cols), generator=g) - 1) * math.sqrt(6 / used_rows)
        parts.append(w.ravel())
    return torch.cat(parts).numpy()


def _guide(bounds, seed, **how):
    guide = guiding.Guide(_ctx(), bounds, **how)
    guide.params = _weights(seed)
    return guide


_BOX = ([-5.0, -5.0, -5.0], [5.0, 5.0, 5.0])


def _film(w, h):
    return torch.zeros((h, w, 8), device="cuda")


def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    if kind == "trace":
        rays = _random_rays(case, seed)
        return {"kind": kind, "mesh": Mesh(ctx, *_icosphere(case["level"])), "rays": rays, "any": case["any_hit"],
                "hits": torch.empty((rays.shape[0], 2), dtype=torch.int32, device="cuda")}
    if kind == "intersect":
        return {"kind": kind, "mesh": Mesh(ctx, *_icosphere(case["level"])), "rays": _camera_rays(case, seed)}
    if kind in ("path", "direct"):
        flat, cam = _flat("cornell")
        t = scenes_guiding.guiding_tracer() if kind == "path" else tracers.DirectLighting()
        return {"kind": kind, "scene": render.GpuScene(ctx, flat), "film": _film(case["width"], case["height"]),
                "desc": render.render_desc(cam, case["width"], case["height"], case["spp"], t, seed=seed + 1)}
    if kind == "guided":
        flat, cam = _flat("slit", case["triangles"])
        guide = _guide(guiding.scene_bounds(flat), seed, guide_probability=0.4, light_probability=0.1)
        return {"kind": kind, "scene": render.GpuScene(ctx, flat), "guide": guide, "film": _film(case["side"], case["side"]),
                "desc": render.render_desc(cam, case["side"], case["side"], case["spp"], scenes_guiding.guiding_tracer(),
                                           seed=seed + 1)}
    if kind == "batch":
        work = _flat("batch", case["scenes"], case["set"], case["triangles"], case["side"], case["spp"])
        t = scenes_batch.batch_tracer()
        entries = [(render.GpuScene(ctx, flat), render.render_desc(w.camera, w.width, w.height, w.spp, t, seed=seed + i))
                   for i, (flat, w) in enumerate(work)]
        return {"kind": kind, "batch": batch.BatchRenderer(ctx, entries, batch.make_config(hero=4))}
    if kind == "photons":
        pos, power, omega, q, normals, r = _photon_inputs(case, seed)
        nq, k = case["queries"], case["k"]
        pmap = photons.PhotonMap(ctx, device_ptr=pos.data_ptr(), n=pos.shape[0], r_max=r, stream=_stream())
        return {"kind": kind, "map": pmap, "pos": pos, "power": power, "omega": omega, "q": q, "normals": normals, "k": k,
                "idx": torch.empty((nq, k), dtype=torch.int32, device="cuda"), "d2": torch.empty((nq, k), device="cuda"),
                "count": torch.empty(nq, dtype=torch.int32, device="cuda"), "xyz": torch.empty((nq, 3), device="cuda")}
    guide = _guide(_BOX, seed)
    rows = case["rows"]
    if kind == "guide_eval":
        return {"kind": kind, "guide": guide, "in": _guide_inputs(rows, seed, False),
                "out": torch.empty((rows, guiding.MIXTURE), device="cuda")}
    return {"kind": kind, "guide": guide, "records": _guide_inputs(rows, seed, True)}


def run(s):
    kind = s["kind"]
    if kind == "trace":
        s["mesh"].trace_into(s["rays"].data_ptr(), s["rays"].shape[0], s["hits"].data_ptr(), s["any"], _stream())
        # which of several occluders an any-hit query reports is left open: only the answer counts
        if s["any"]:
            return {"hit": s["hits"][:, 0] >= 0}
        return {"prim": s["hits"][:, 0], "t": s["hits"][:, 1].view(torch.float32)}
    if kind == "intersect":
        prim, t = s["mesh"].intersect(s["rays"])
        return {"prim": prim, "t": t}
    if kind in ("path", "direct"):
        s["film"].zero_()
        s["scene"].render_device(s["desc"], s["film"].data_ptr(), _stream())
        return s["film"]
    if kind == "guided":
        s["film"].zero_()
        s["guide"].render(s["scene"], s["desc"], s["film"].data_ptr(), train=False)
        return s["film"]
    if kind == "batch":
        s["batch"].reset_films()
        s["batch"].launch(_stream())
        return s["batch"].films
    if kind == "photons":
        m, ctx, st = s["map"], s["map"].ctx, _stream()
        m.rebuild(s["pos"].data_ptr(), s["pos"].shape[0], stream=st)
        nq = s["q"].shape[0]
        m.gather_device(s["q"].data_ptr(), nq, s["k"], s["idx"].data_ptr(), s["d2"].data_ptr(), s["count"].data_ptr(), st)
        ctx.check(ctx._lib.liar_gpu_photon_estimate_device(
            ctx.handle, s["power"].data_ptr(), s["omega"].data_ptr(), s["pos"].shape[0], s["normals"].data_ptr(), nq,
            s["k"], s["idx"].data_ptr(), s["d2"].data_ptr(), s["count"].data_ptr(), C.c_float(1.0 / s["pos"].shape[0]),
            s["xyz"].data_ptr(), C.c_void_p(st)))
        return {"idx": s["idx"], "d2": s["d2"], "count": s["count"], "xyz": s["xyz"]}
    if kind == "guide_eval":
        return s["guide"].eval(s["in"], out=s["out"])
    loss, grad = s["guide"].train_step(s["records"], apply=True, want_grad=True)
    return {"loss": loss, "grad": grad}


# ---- what a pass cannot do without

_NET = 225 * 64 + 4 * 64 * 64 + 64 * 40  # multiply-adds of the network for one row


def work(case):
    kind = case["kind"]
    if kind in ("trace", "intersect"):
        n = case["rays"] if kind == "trace" else case["width"] * case["height"]
        # a ray in and its hit out; of the model, at most the triangles there are (36 bytes each); one
        # exact intersection test (about 50 operations) and a box test (about 25) per tree level
        tris = 20 * 4 ** case["level"]
        return {"bytes": 40 * n + 36 * min(tris, n), "flops": n * (50 + 25 * math.log2(tris))}
    if kind in ("path", "direct", "guided"):
        w, h = (case["side"],) * 2 if kind == "guided" else (case["width"], case["height"])
        # the film's sums once; about 2.5 segments a path or 32 shadow rays a sample, 500 operations each
        paths = w * h * case["spp"]
        segments = {"path": 2.5, "direct": 33, "guided": 3}[kind] * paths
        net = 2 * _NET * paths if kind == "guided" else 0
        return {"bytes": 32 * w * h + (36 * case["triangles"] if kind == "guided" else 0), "flops": 500 * segments + net}
    if kind == "batch":
        params = scenes_batch.batch_workload_params(case["scenes"], case["set"], (10000, case["triangles"]),
                                                    (64, case["side"]), (2, case["spp"]))
        return {"bytes": sum(36 * t + 32 * s * s for _, t, s, _ in params),
                "flops": sum(500 * 1.6 * s * s * p for _, _, s, p in params)}
    if kind == "photons":
        n, nq, k = case["photons"], case["queries"], case["k"]
        return {"bytes": 12 * n + nq * (12 + 12 + 8 * k + 4 + 12) + 24 * min(n, nq * k), "flops": nq * k * 18}
    n = case["rows"]
    if kind == "guide_eval":
        return {"bytes": n * 4 * (9 + 40), "flops": 2 * _NET * n}
    return {"bytes": n * 4 * 13, "flops": 6 * _NET * n}


# ---- the same in 64 bits


def _closest(v, f, rays):
    """t of the nearest triangle along each ray (Moller and Trumbore 1997), inf for none."""
    v = torch.from_numpy(v).cuda().double()
    f = torch.from_numpy(f.astype(np.int64)).cuda()
    a, e1, e2 = v[f[:, 0]], v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]]
    n = torch.cross(e1, e2, dim=1)
    out = []
    step = max(1, int(2e8 // len(f)))
    for r in rays.double().split(step):
        o, d = r[:, 0:3], r[:, 4:7]
        # det = -d . n; the numerators are linear in (o, d) through the Pluecker moment m = o x d
        m = torch.cross(o, d, dim=1)
        det = -(d @ n.T)
        u = (m @ e2.T) + d @ torch.cross(a, e2, dim=1).T
        w = -(m @ e1.T) - d @ torch.cross(a, e1, dim=1).T
        t = o @ n.T - (a * n).sum(1)
        u, w, t = u / det, w / det, t / det
        t[~((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0))] = math.inf
        out.append(t.min(1).values)
    return torch.cat(out)


def _neighbours(pos, q, k, r):
    """(squared distances ascending, indices) of the k photons nearest to each query within r."""
    p = pos.double()
    ds, ix = [], []
    for c in q.double().split(max(1, int(4e8 // len(p)))):
        d = sum((c[:, None, a] - p[None, :, a]) ** 2 for a in range(3))
        d, i = d.topk(min(k, len(p)), dim=1, largest=False, sorted=True)
        ds.append(d)
        ix.append(i)
    d, i = torch.cat(ds), torch.cat(ix)
    out = d >= float(np.float32(r) * np.float32(r))
    d[out] = math.inf
    return d, i, (~out).sum(1)


def _network(params, x):
    """The raw outputs (n, 48) of the guide network for normalised inputs x (n, 9)."""
    freq = math.pi * 2.0 ** (0.5 * torch.arange(12, device="cuda", dtype=torch.float64))
    a = x[:, :, None] * freq
    h = torch.stack([a.sin(), a.cos()], 3).reshape(len(x), 216)
    h = torch.cat([h, x, x.new_zeros(len(x), 31)], 1)
    at = 0
    for rows, cols in ((256, 64), (64, 64), (64, 64), (64, 64), (64, 64), (64, 48)):
        h = h @ params[at:at + rows * cols].view(rows, cols)
        at += rows * cols
        h = h.relu() if cols == 64 else h
    return h


def _lobes(o):
    o = o[:, :40].reshape(-1, 8, 5)
    m = o[..., 0:3]
    return m / m.norm(dim=2, keepdim=True), o[..., 3].clamp(-6, 7).exp(), o[..., 4].softmax(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace":
        if case["any_hit"] or case["rays"] * 20.0 * 4 ** case["level"] > PAIRS:
            return None
        return {"prim": None, "t": _closest(*_icosphere(case["level"]), _random_rays(case, seed))}
    if kind == "intersect":
        if case["width"] * case["height"] * 20.0 * 4 ** case["level"] > PAIRS:
            return None
        t = _closest(*_icosphere(case["level"]), torch.from_numpy(_camera_rays(case, seed)).cuda())
        return {"prim": None, "t": t.cpu().numpy()}
    if kind == "photons":
        if float(case["photons"]) * case["queries"] > PAIRS:
            return None
        pos, power, omega, q, normals, r = _photon_inputs(case, seed)
        d, i, c = _neighbours(pos, q, case["k"], r)
        use = d.isfinite() & ((omega.double()[i] * normals.double()[:, None]).sum(2) > 0)
        xyz = (power.double()[i] * use[..., None]).sum(1) / len(pos)
        far = torch.where(d.isfinite(), d, -1.0).max(1).values
        xyz = torch.where((far > 0)[:, None], xyz / (math.pi * far[:, None]), 0.0)
        return {"idx": None, "d2": d, "count": None, "xyz": xyz}
    if kind not in ("guide_eval", "guide_train"):
        return None  # Monte Carlo images: the sum over the renderer's own samples has no closed form
    params = torch.from_numpy(_weights(seed)).cuda().double()
    rec = _guide_inputs(case["rows"], seed, kind == "guide_train").double()
    rec[:, 0:3] = (rec[:, 0:3] + 5) / 10
    if kind == "guide_eval":
        out = []
        for x in rec.split(1 << 18):
            mu, kappa, pi = _lobes(_network(params, x))
            out.append(torch.cat([torch.cat([mu, kappa[..., None]], 2).reshape(-1, 32), pi], 1))
        return torch.cat(out)
    # negative log density of the sampled directions, weights over their mean clipped at 20
    params.requires_grad_(True)
    mu, kappa, pi = _lobes(_network(params, rec[:, :9]))
    cos = (mu * rec[:, None, 9:12]).sum(2)
    log = (kappa / -torch.expm1(-2 * kappa)).log() - math.log(2 * math.pi) + kappa * (cos - 1)
    w = (rec[:, 12] / rec[:, 12].mean()).clamp(max=20)
    loss = -(w * (pi.log() + log).logsumexp(1)).mean()
    loss.backward()
    return {"loss": float(loss), "grad": params.grad.cpu().numpy()}
