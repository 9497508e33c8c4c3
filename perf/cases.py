"""The work this renderer is measured by: render calls of every public form
(whole images, device films, batches of views on the device and to the host,
the serving loop), ray queries and BSDF batches, over the sizes that callers
use, from a thumbnail of some thousand paths to views of tens of millions.

listed() gives the cases, draw(rng) more of the same ranges.  prepare() makes
what a caller holds before the call (a resident scene, films, rays, records, a
server with its scenes), run() is one pass through the public entry points,
work() the bytes and operations that the pass cannot do without, and exact()
its outputs in 64 bits where they have a closed form.
"""
import atexit
import math
import weakref

import numpy as np
import torch

import hikari_b200 as hk
from hikari_b200 import scenes, serving
from hikari_b200.scenedesc import BECKMANN

# The launch configuration that the benchmark's autotuner settles on for the
# heterogeneous scene: a caller who renders many views of one scene tunes once
# and passes it with every batch.
TUNED = dict(capacity=1 << 22, threads_extend=128, threads_shade=64, iterations_per_check=16, fetch_steps=6,
             fetch_min_idle=8, fetch_steps_shadow=3, fetch_min_idle_shadow=8, shadow_tests=2, closest_tests=2)

# Triangles and rays per path (closest-hit + shadow, as the renderer's own
# counters give them) of the scenes below.
SCENES = {
    "cornell": (36, 18.0),             # diffuse Cornell box, one area light
    "smooth": (40, 16.0),              # Cornell box of delta, two-sided and coated materials
    "heterogeneous": (1.36e6, 5.8),    # 64 displaced spheres, six rough materials, 4 area lights + sky
    "mesh_conductor": (327682, 4.0),   # one displaced sphere of 327,680 triangles on a ground quad under the sky
    "mesh_dielectric": (327682, 7.0),
    "mesh_plastic": (327682, 4.5),
    "textured": (1612, 8.0),           # bitmap, procedural, bump and normal maps; every emitter kind
}
MATERIALS = {name: desc for name, desc in scenes.config2_materials()}
OUTPUT_FLOPS = {"conductor": 260.0, "dielectric": 300.0, "plastic": 400.0, "coated": 900.0}   # per BSDF record


def listed():
    return [
        # the smallest call: a thumbnail while a scene is being set up; latency counts
        {"name": "thumbnail", "kind": "image", "scene": "cornell", "width": 64, "height": 64, "spp": 4, "depth": 16},
        # the plain small benchmark image, 2^22 paths of up to 64 bounces
        {"name": "cornell", "kind": "image", "scene": "cornell", "width": 256, "height": 256, "spp": 64, "depth": 64},
        # a quick look at a large scene: an odd-sized still of a million paths
        {"name": "still", "kind": "image", "scene": "heterogeneous", "width": 501, "height": 283, "spp": 8, "depth": 16},
        # an ordinary still of one heavy mesh with transmission
        {"name": "glass", "kind": "image", "scene": "mesh_dielectric", "width": 512, "height": 512, "spp": 32, "depth": 16},
        # views of a large scene with a tuned configuration, films kept on the device: the largest case
        {"name": "views", "kind": "batch", "scene": "heterogeneous", "width": 1024, "height": 1024, "spp": 32, "depth": 16,
         "views": 2, "tuned": True},
        # a handful of views of odd and different sizes with the default configuration
        {"name": "views_odd", "kind": "batch", "scene": "heterogeneous", "width": 383, "height": 217, "spp": 16, "depth": 16,
         "views": 5, "tuned": False},
        # textured views delivered to host memory
        {"name": "textured", "kind": "batch_host", "scene": "textured", "width": 512, "height": 512, "spp": 16, "depth": 12,
         "views": 2},
        # one pass of samples into a film that the caller keeps on the device (asynchronous call)
        {"name": "film", "kind": "film", "scene": "smooth", "width": 200, "height": 150, "spp": 16, "depth": 32},
        # closest-hit queries against a mesh: picking, baking, ambient visibility
        {"name": "rays", "kind": "trace", "scene": "mesh_plastic", "n": 1000003, "any_hit": False},
        # a small batch of closest-hit queries against a room
        {"name": "rays_room", "kind": "trace", "scene": "cornell", "n": 65536, "any_hit": False},
        # sample, eval and pdf of one material over a record array
        {"name": "bsdf", "kind": "bsdf", "material": "conductor_ggx_cu_a0.2", "n": 1 << 22},
        # jobs of several sizes and scenes submitted together to the serving loop
        {"name": "serving", "kind": "serve", "jobs": 9, "side": 160, "spp": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image", "image", "image", "batch", "batch", "batch_host", "film", "trace", "bsdf", "serve"])
    if kind == "trace":
        return {"kind": kind, "scene": rng.choice(["cornell", "mesh_plastic", "mesh_conductor", "heterogeneous"]),
                "n": _log(rng, 1 << 14, 1 << 21), "any_hit": rng.random() < 0.4}
    if kind == "bsdf":
        return {"kind": kind, "material": rng.choice(sorted(MATERIALS)), "n": _log(rng, 1 << 14, 1 << 23)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(3, 16), "side": _log(rng, 64, 256), "spp": _log(rng, 8, 64)}
    scene = rng.choice(["cornell", "smooth", "textured"] if kind == "film" else sorted(SCENES))
    views = rng.randint(1, 6) if kind in ("batch", "batch_host") else 1
    limit = (1 << 20) if kind == "film" else (1 << 24)    # paths of a drawn call
    width = _log(rng, 48, 400 if kind == "film" else 1100)
    height = max(32, int(width * rng.uniform(0.5, 1.2)))
    spp = max(1, min(_log(rng, 1, 64), limit // (width * height * views)))
    case = {"kind": kind, "scene": scene, "width": width, "height": height, "spp": spp, "depth": rng.choice([8, 16, 32])}
    if kind in ("batch", "batch_host"):
        case["views"] = views
    if kind == "batch":
        case["tuned"] = width * height * spp * views >= (1 << 23) and rng.random() < 0.5
    return case


def _scene(name, seed, width, height, depth):
    if name == "cornell":
        return scenes.cornell_box(seed=seed, width=width, height=height, depth=depth)
    if name == "smooth":
        return scenes.cornell_smooth(seed=seed, width=width, height=height, depth=depth)
    if name == "textured":
        return scenes.lights_scene(width=width, height=height, depth=depth, seed=seed, shading_normals=True, textured=True,
                                   bitmap=True, bump=True)
    if name == "heterogeneous":
        return scenes.heterogeneous(width=width, height=height, depth=depth, levels=(4, 5, 6), env_res=(1024, 512), seed=seed)
    return scenes.mesh_heavy(name.split("_")[1], width=width, height=height, depth=depth, level=7, env_res=(1024, 512),
                             seed=seed)


def _poses(name, n, seed):
    """Camera poses of n views: around the heterogeneous scene, elsewhere the scene's own camera (None)."""
    if name != "heterogeneous":
        return [None] * n
    out = []
    for k in range(n):
        a = 2 * math.pi * (k / n + (seed % 97) / 97.0)
        out.append(scenes.look_at((42 * math.sin(a), 18, 42 * math.cos(a)), (0, 3, 0), (0, 1, 0)))
    return out


def _sizes(case):
    """Image sizes of a batch: the case's size, views after the first a little smaller where it is untuned."""
    shrink = 0 if case.get("tuned", True) else 29
    return [(max(32, case["width"] - shrink * k), max(32, case["height"] - shrink * k // 2)) for k in range(case["views"])]


def _rays(case, seed):
    """Rays from points around the scene towards points inside it, with the renderer's epsilon as mint."""
    g = torch.Generator().manual_seed(seed + 1)
    n, name = case["n"], case["scene"]
    centre, inner, outer = {"cornell": ((0.0, 1.0, 0.0), 0.9, 0.9), "heterogeneous": ((0.0, 5.0, 0.0), 18.0, 40.0)}.get(
        name, ((0.0, 1.0, 0.0), 1.0, 3.0))
    c = torch.tensor(centre)
    to = c + inner * (2 * torch.rand(n, 3, generator=g) - 1)
    fr = c + outer * (2 * torch.rand(n, 3, generator=g) - 1)
    d = to - fr
    rays = torch.empty(n, 8)
    rays[:, 0:3] = fr
    rays[:, 6] = 1e-4
    if case["any_hit"]:     # a visibility query: the segment between the two points
        rays[:, 3:6], rays[:, 7] = d, 1.0 - 1e-4
    else:
        rays[:, 3:6], rays[:, 7] = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6), math.inf
    return rays


def _records(case, seed):
    """Records of a BSDF batch: directions over the upper hemisphere (dielectrics: the sphere) and uniform samples."""
    g = torch.Generator().manual_seed(seed + 1)
    n = case["n"]

    def directions(lo):
        z = lo + (1 - lo) * torch.rand(n, generator=g)
        p = 2 * math.pi * torch.rand(n, generator=g)
        s = (1 - z * z).clamp_min(0).sqrt()
        return torch.stack([s * p.cos(), s * p.sin(), z], 1).contiguous()

    lo = -1.0 if case["material"].startswith("dielectric") else 1e-3
    wi, wo = directions(lo), directions(lo)
    return wi, torch.rand(n, 2, generator=g), torch.rand(n, generator=g), wo


# servers that still run are closed before the interpreter takes the device down
_servers = weakref.WeakSet()


@atexit.register
def _close_servers():
    for s in list(_servers):
        s.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        sd = _scene(case["scene"], seed, 64, 64, 8)
        return {"case": case, "scene": hk.Scene.from_desc(sd), "rays": _rays(case, seed).cuda()}
    if kind == "bsdf":
        sc = hk.Scene.from_desc(scenes.bsdf_scene([(case["material"], MATERIALS[case["material"]])]))
        wi, u2, u1, wo = (t.cuda() for t in _records(case, seed))
        return {"case": case, "scene": sc, "id": 0, "wi": wi, "u2": u2, "u1": u1, "wo": wo}
    if kind == "serve":
        side = case["side"]
        sds = [_scene(s, seed, side, side, 16) for s in ("cornell", "smooth", "mesh_plastic")]
        held = [hk.Scene.from_desc(sd) for sd in sds]
        server = serving.Server(capacity=1 << 18, hbm_budget=4 << 30)
        _servers.add(server)
        jobs = []
        for k in range(case["jobs"]):
            w, h = max(32, side - 11 * k), max(32, side - 7 * k)
            out = torch.empty((h, w, 3), pin_memory=True).numpy()
            jobs.append(dict(scene=k % 3, spp=max(1, case["spp"] >> (k % 2)), seed=seed * 64 + k, width=w, height=h, out=out))
        return {"case": case, "server": server, "ids": [server.add_scene(s) for s in held], "jobs": jobs}
    sd = _scene(case["scene"], seed, case["width"], case["height"], case["depth"])
    scene = hk.Scene.from_desc(sd)
    state = {"case": case, "scene": scene, "seed": seed}
    if kind == "image":
        state["out"] = torch.empty((case["height"], case["width"], 3), pin_memory=True).numpy()
    elif kind == "film":
        state["film"] = torch.zeros(scene.film_shape(), device="cuda")
    else:
        state["cameras"] = _poses(case["scene"], case["views"], seed)
        if kind == "batch":
            state["sizes"] = _sizes(case)
            state["films"] = [torch.zeros(scene.film_shape(w, h), device="cuda") for w, h in state["sizes"]]
        else:
            state["outs"] = [torch.empty((case["height"], case["width"], 3), pin_memory=True).numpy()
                             for _ in range(case["views"])]
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "trace":
        tri, t, u, v, _ = state["scene"].trace(state["rays"], any_hit=case["any_hit"])
        return tri if case["any_hit"] else (tri, t, u, v)
    if kind == "bsdf":
        return state["scene"].bsdf_batch(state["id"], state["wi"], state["u2"], state["u1"], state["wo"])
    if kind == "serve":
        srv, handles, images = state["server"], [], []
        for j in state["jobs"]:
            jid, out = srv.submit(state["ids"][j["scene"]], j["spp"], 16, j["seed"], j["width"], j["height"], out=j["out"])
            handles.append(jid)
            images.append(out)
        for jid in handles:
            srv.wait(jid)
        return images
    scene, seed, spp, depth = state["scene"], state["seed"], case["spp"], case["depth"]
    if kind == "image":
        img, _ = scene.render_image(spp, depth, seed, out=state["out"])
        return img
    if kind == "film":
        state["film"].zero_()
        scene.render(state["film"], spp, depth, seed)
        return state["film"]
    seeds = [seed * 16 + k for k in range(case["views"])]
    if kind == "batch":
        for f in state["films"]:
            f.zero_()
        scene.render_batch(state["films"], spp, depth, seeds=seeds, cameras=state["cameras"], sizes=state["sizes"],
                           **(TUNED if case["tuned"] else {}))
        return state["films"]
    scene.render_batch_host(state["outs"], spp, depth, seeds=seeds, cameras=state["cameras"])
    return state["outs"]


def work(case):
    """Each input read once, each output written once; the operations of a ray
    are about nine visits of eight boxes (18 operations a box) and four
    triangle tests of 60, those of a path vertex about 400."""
    kind = case["kind"]
    if kind == "bsdf":
        return {"bytes": 84.0 * case["n"], "flops": OUTPUT_FLOPS[case["material"].split("_")[0]] * case["n"]}
    per_ray = 9 * 8 * 18 + 4 * 60
    if kind == "trace":
        tris, _ = SCENES[case["scene"]]
        return {"bytes": case["n"] * (32.0 + (4 if case["any_hit"] else 16)) + 55.0 * tris, "flops": float(per_ray) * case["n"]}
    if kind == "serve":
        paths = pixels = 0
        for k in range(case["jobs"]):
            px = max(32, case["side"] - 11 * k) * max(32, case["side"] - 7 * k)
            pixels += px
            paths += px * max(1, case["spp"] >> (k % 2))
        tris, rays = 328000.0, 13.0
    else:
        tris, rays = SCENES[case["scene"]]
        if kind == "batch":
            pixels = sum(w * h for w, h in _sizes(case))
        else:
            pixels = case["width"] * case["height"] * case.get("views", 1)
        paths = pixels * case["spp"]
    return {"bytes": 55.0 * tris + 16.0 * pixels, "flops": paths * rays * (per_ray + 200.0)}


# ------------------------------------------------------------ outputs in 64 bits
def _exact_conductor(case, seed):
    """The GGX / Beckmann rough conductor's sampled direction, weight and pdf,
    and eval and pdf of the given directions (src/bsdf/RoughConductorBSDF.cpp:54-154,
    src/core/MicrofacetDistribution.cpp:34-240), for isotropic roughness."""
    m = MATERIALS[case["material"]]
    wi, u2, _, wo = (t.cuda().double() for t in _records(case, seed))
    a = float(np.float32(m.alpha_u))
    eta = torch.tensor(np.float32(m.conductor_eta()).astype(np.float64), device="cuda")
    k = torch.tensor(np.float32(m.k).astype(np.float64), device="cuda")
    ks = torch.tensor(np.float32(m.ks).astype(np.float64), device="cuda")

    def distribution(h):
        c2 = h[:, 2] ** 2
        be = (h[:, 0] ** 2 + h[:, 1] ** 2) / (a * a) / c2
        if m.distribution == BECKMANN:
            r = torch.exp(-be) / (math.pi * a * a * c2 * c2)
        else:
            r = 1.0 / (math.pi * a * a * ((1 + be) * c2) ** 2)
        return torch.where((h[:, 2] <= 0) | (r * h[:, 2] < 1e-20), torch.zeros_like(r), r)

    def g1(v, h):
        root = a * (1 - v[:, 2] ** 2).clamp_min(0).sqrt() / v[:, 2].abs()
        if m.distribution == BECKMANN:
            x = 1.0 / root
            g = torch.where(x >= 1.6, torch.ones_like(x), (3.535 * x + 2.181 * x * x) / (1 + 2.276 * x + 2.577 * x * x))
        else:
            g = 2.0 / (1 + (1 + root * root).sqrt())
        return torch.where((v * h).sum(1) * v[:, 2] <= 0, torch.zeros_like(g), g)

    def fresnel(c):
        c2 = (c * c)[:, None]
        s2 = 1 - c2
        t0 = eta * eta - k * k - s2
        ab = (t0 * t0 + 4 * eta * eta * k * k).sqrt()
        t1, t2 = ab + c2, 2 * c[:, None] * (0.5 * (ab + t0)).sqrt()
        rs = (t1 - t2) / (t1 + t2)
        t3, t4 = c2 * ab + s2 * s2, t2 * s2
        return 0.5 * (rs * (t3 - t4) / (t3 + t4) + rs)

    zero = torch.zeros_like(wi[:, 0])
    # the given directions
    h = wi + wo
    h = h / h.norm(dim=1, keepdim=True)
    d = distribution(h)
    e_rgb = (d * g1(wi, h) * g1(wo, h) / (4 * wi[:, 2]))[:, None] * fresnel((h * wi).sum(1)) * ks
    ok = (wi[:, 2] > 0) & (wo[:, 2] > 0)
    e_rgb = torch.where((ok & (d != 0))[:, None], e_rgb, torch.zeros_like(e_rgb))
    p_pdf = torch.where(ok, d * h[:, 2] / (4 * (h * wo).sum(1).abs()), zero)
    # the sampled direction
    ph = 2 * math.pi * u2[:, 1]
    t2 = a * a * (-torch.log1p(-u2[:, 0]) if m.distribution == BECKMANN else u2[:, 0] / (1 - u2[:, 0]))
    cm = 1.0 / (1 + t2).sqrt()
    sm = (1 - cm * cm).clamp_min(0).sqrt()
    h = torch.stack([sm * ph.cos(), sm * ph.sin(), cm], 1)
    mdw = (h * wi).sum(1)
    s_wo = 2 * mdw[:, None] * h - wi
    d = distribution(h)
    w = (d * g1(wi, h) * g1(s_wo, h) * mdw / (d * cm * wi[:, 2]))[:, None] * fresnel(mdw) * ks
    keep = (wi[:, 2] > 0) & (s_wo[:, 2] >= 0)
    w = torch.where(keep[:, None], w, torch.zeros_like(w))
    s_pdf = torch.where(keep & (s_wo[:, 2] > 0) & (w != 0).any(1), d * cm / (4 * (h * s_wo).sum(1).abs()), zero)
    return dict(s_wo=s_wo, s_w=w, s_pdf=s_pdf, s_measure=None, e_rgb=e_rgb, p_pdf=p_pdf)


def _exact_room(case, seed):
    """Distance to the nearest triangle of a small scene by testing them all;
    the triangle and its barycentrics are left out, as where two triangles of
    the room meet either one is right."""
    sd = _scene(case["scene"], seed, 64, 64, 8)
    P = torch.tensor(np.concatenate([m.positions[m.indices] for m in sd.meshes]), device="cuda").double()
    rays = _rays(case, seed).cuda().double()
    o, d = rays[:, 0:3], rays[:, 3:6]
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device="cuda")
    for p0, p1, p2 in P:
        e1, e2 = p1 - p0, p2 - p0
        pv = torch.linalg.cross(d, e2.expand_as(d))
        det = pv @ e1
        tv = o - p0
        qv = torch.linalg.cross(tv, e1.expand_as(d))
        u, v, t = (tv * pv).sum(1) / det, (qv * d).sum(1) / det, (qv @ e2) / det
        hit = (det.abs() >= 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= rays[:, 6]) & (t <= best)
        best = torch.where(hit, t, best)
    t = torch.where(torch.isinf(best), torch.zeros_like(best), best)
    return None, t, None, None


def exact(case, seed):
    """Images are Monte Carlo sums over millions of branching paths: they have
    no closed form, and a 64-bit path tracer follows other paths."""
    if case["kind"] == "bsdf" and case["material"].startswith("conductor"):
        return _exact_conductor(case, seed)
    if case["kind"] == "trace" and case["scene"] == "cornell" and not case["any_hit"]:
        return _exact_room(case, seed)
    return None
