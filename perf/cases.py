"""What users of this framework have it do, as cases to be timed: ray queries, renders and the
path-guiding network's training pass, each through the package's public entry points.

A case is a dict of plain values; "kind" names the entry point, the rest its sizes. Geometry
belongs to the case (a program keeps its scene and asks for many frames or rays of it), the rays,
samples and training rows to the seed. The exception is "scene_edit", whose scene is the seed's:
there every pass brings a scene the device does not hold.

  rays        Accel.trace_device: rays and hits in device memory, the BVH handle kept
  rays_host   Accel.trace_host: rays and hits in pinned host memory (a renderer that is not this one)
  v4          render_v4 (prgpu_render): the drop-in float film of PRender's GPU module
  render      render_ex (prgpu_render_ex): FP64 film, with the box family's media, occluder or light BVH
  scene_edit  render_ex on a scene that changed since the last call
  outdoor     render_ex on the terrain / cloud / metal-sphere scene under sun and sky
  guided      render_ex sampling with the guide network
  batch       render_batch: several renders of uneven size in one graph launch
  train       guide.gradient: loss and weight gradients of a batch of training rows
"""

import functools
import math
import os
import sys

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ar-renderer_b200"))

import numpy as np  # noqa: E402
import torch  # noqa: E402

from prgpu import abi, guide, hostscene, render, scenes, trace, workloads  # noqa: E402


def listed():
    return [
        # A picking or probe query: a few thousand rays at a small mesh; latency of one launch.
        {"name": "rays_probe", "kind": "rays", "tris": 4096, "leaf": 4, "rays": 4096, "any": False, "seed0": 1},
        # Visibility of an image's worth of samples (odd count) in a mid-sized mesh.
        {"name": "rays_visibility", "kind": "rays", "tris": 100003, "leaf": 4, "rays": 1500007, "any": True, "seed0": 2},
        # The traversal microbenchmark's closest-hit pass, at its own size.
        {"name": "rays_closest_16m", "kind": "rays", "tris": 1 << 20, "leaf": 1, "rays": 1 << 24, "any": False,
         "seed0": 1},
        # Rays of another program, host memory to host memory.
        {"name": "rays_from_host", "kind": "rays_host", "tris": 100003, "leaf": 4, "rays": 2000003, "any": False,
         "seed0": 3},
        # An interactive preview: one sample per pixel of a thumbnail, depth 8.
        {"name": "preview", "kind": "v4", "w": 64, "h": 64, "spp": 1, "depth": 8, "seed0": 0},
        # The same after an edit of the scene: validation, conversion and upload inside the call.
        {"name": "scene_edit", "kind": "scene_edit", "w": 160, "h": 90, "spp": 4, "depth": 8},
        # The plain path tracer's benchmark scene and settings.
        {"name": "box_64spp", "kind": "render", "w": 256, "h": 256, "spp": 64, "depth": 8, "medium": False,
         "slit": False, "light_bvh": False, "seed0": 0},
        # The box filled with the chromatic medium, light-BVH sampling, a ragged film, longer paths.
        {"name": "fog_16spp", "kind": "render", "w": 317, "h": 181, "spp": 16, "depth": 16, "medium": True,
         "slit": False, "light_bvh": True, "seed0": 4},
        # The outdoor scene: terrain, cloud grid, analytic metal spheres, sun and sky, depth 64.
        {"name": "outdoor_8spp", "kind": "outdoor", "w": 480, "h": 270, "spp": 8, "depth": 64, "terrain": 512,
         "cloud": 64, "spheres": 40},
        # The slit scene with its subsurface spheres, diffuse vertices sampled with the guide network.
        {"name": "guided_slit", "kind": "guided", "w": 128, "h": 128, "spp": 32, "depth": 32, "seed0": 0},
        # Six renders of the uneven batch (128^2 .. 1024^2, half with media) at 1/16 of their samples.
        {"name": "batch_uneven", "kind": "batch", "first": 0, "count": 6, "div": 16},
        # One training batch of the guide network at the size the renderer trains with.
        {"name": "guide_train_64k", "kind": "train", "rows": 1 << 16},
    ]


def _between(rng, lo, hi):
    """Spread over the logarithm of the range, odd sizes among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "rays_host", "v4", "scene_edit", "render", "render", "outdoor", "guided",
                       "batch", "train"])
    if kind == "rays":
        return {"kind": kind, "tris": _between(rng, 500, 1 << 20), "leaf": rng.choice([1, 2, 4]),
                "rays": _between(rng, 1000, 1 << 23), "any": rng.random() < 0.5, "seed0": rng.randrange(1000)}
    if kind == "rays_host":
        return {"kind": kind, "tris": _between(rng, 500, 1 << 18), "leaf": rng.choice([1, 2, 4]),
                "rays": _between(rng, 1000, 1 << 22), "any": rng.random() < 0.5, "seed0": rng.randrange(1000)}
    if kind == "v4":
        return {"kind": kind, "w": _between(rng, 32, 400), "h": _between(rng, 32, 400), "spp": rng.choice([1, 2, 4]),
                "depth": rng.choice([4, 8, 16]), "seed0": rng.randrange(1000)}
    if kind == "scene_edit":
        return {"kind": kind, "w": _between(rng, 64, 320), "h": _between(rng, 64, 320), "spp": rng.choice([1, 4]),
                "depth": rng.choice([4, 8])}
    if kind == "render":
        return {"kind": kind, "w": _between(rng, 64, 512), "h": _between(rng, 64, 512), "spp": _between(rng, 8, 24),
                "depth": rng.choice([8, 16, 32]), "medium": rng.random() < 0.5, "slit": rng.random() < 0.3,
                "light_bvh": rng.random() < 0.5, "seed0": rng.randrange(1000)}
    if kind == "outdoor":
        return {"kind": kind, "w": _between(rng, 100, 640), "h": _between(rng, 100, 360), "spp": _between(rng, 4, 12),
                "depth": rng.choice([16, 64]), "terrain": _between(rng, 64, 512), "cloud": rng.choice([16, 33, 64]),
                "spheres": rng.choice([1, 40, 200])}
    if kind == "guided":
        return {"kind": kind, "w": _between(rng, 64, 200), "h": _between(rng, 64, 200), "spp": _between(rng, 8, 32),
                "depth": rng.choice([16, 32]), "seed0": rng.randrange(1000)}
    if kind == "batch":
        return {"kind": kind, "first": rng.randrange(40), "count": rng.choice([2, 3, 5, 8]), "div": rng.choice([16, 32])}
    return {"kind": "train", "rows": _between(rng, 1000, 1 << 16)}


# ---------------------------------------------------------------------------------------------
# Geometry (the case's) and per-seed inputs


@functools.lru_cache(maxsize=6)
def _soup(tris, leaf, seed0):
    """Triangles of the microbenchmark's soup at its own density, and the host library's BVH."""
    verts = workloads.triangle_soup(tris, seed=seed0, edge=0.01 * ((1 << 20) / tris) ** (1 / 3))
    nodes, order = trace.build_bvh_triangles(verts, max_leaf=leaf)
    return verts, nodes, order


def _rays(n, any_hit, seed):
    """(n, 8) float32 on the device, in the layout of prgpu::Ray: o, tMax, d, pad. Origins uniform
    in [-0.5, 1.5]^3, directions uniform on the sphere, tMax infinite or uniform in [0, 2]."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = torch.zeros((n, 8), device="cuda")
    r[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 0.5
    r[:, 3] = torch.rand(n, generator=g, device="cuda") * 2.0 if any_hit else math.inf
    z = 1.0 - 2.0 * torch.rand(n, generator=g, device="cuda")
    s = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    phi = 2.0 * math.pi * torch.rand(n, generator=g, device="cuda")
    r[:, 4], r[:, 5], r[:, 6] = s * torch.cos(phi), s * torch.sin(phi), z
    return r


@functools.lru_cache(maxsize=4)
def _box(seed0, w, h, medium, slit, light_bvh):
    s = scenes.slit_scene(seed=seed0, width=w, height=h) if slit else scenes.box_scene(seed=seed0, width=w, height=h)
    if medium:
        s.medium = scenes.box_scene(seed=seed0, medium=True, subdiv=0).medium
    hs = hostscene.build_box_scene(s)
    lights = hs.light_bvh() if light_bvh else None
    return hs, render.make_ext(light_bvh=lights)


@functools.lru_cache(maxsize=2)
def _outdoor(w, h, terrain, cloud, spheres):
    return hostscene.build_large_scene(w, h, terrain_res=terrain, cloud_res=cloud, spheres=spheres, sky_resolution=256)


@functools.lru_cache(maxsize=2)
def _batch(first, count, div):
    specs = scenes.uneven_batch(48)[first:first + count]
    return [(hostscene.build_box_scene(s), max(1, s.spp // div), s.max_depth, s.height, s.width) for s in specs]


@functools.lru_cache(maxsize=1)
def _guide_weights():
    """He-uniform weights with the network's constant units kept: the bias columns start at zero,
    no weight leads into a constant unit or an unused output."""
    rng = np.random.default_rng(12)
    parts = []
    for rows, cols, layer in ((64, 128, 0), (64, 64, 1), (64, 64, 2), (64, 64, 3), (48, 64, 4)):
        used = 81 if layer == 0 else 63
        m = np.zeros((rows, cols))
        live = 41 if layer == 4 else 63
        lim = math.sqrt(6.0 / (82 if layer == 0 else cols))
        m[:live, :used] = rng.uniform(-lim, lim, (live, used))
        parts.append(m.ravel())
    return np.concatenate(parts).astype(np.float32)


def _train_rows(rows, seed):
    """Training rows as the renderer records them: positions in the unit cube (12-band encoding),
    unit normals and directions, wi on the side of n that wo is on, a cosine BSDF pdf, and
    radiance weights spread like a path tracer's (log-normal, mean about 1)."""
    rng = np.random.default_rng(seed)
    unit = lambda v: v / np.linalg.norm(v, axis=1, keepdims=True)  # noqa: E731
    x = rng.random((rows, 3))
    n, wo, wi = (unit(rng.normal(size=(rows, 3))) for _ in range(3))
    wo *= np.sign((wo * n).sum(1, keepdims=True))
    wi *= np.sign((wi * n).sum(1, keepdims=True))
    f = np.zeros((rows, 128), np.float32)
    f[:, 0:3] = x
    for b in range(12):
        f[:, 3 + 6 * b:9 + 6 * b:2] = np.sin(math.pi * x * 2.0 ** b)
        f[:, 4 + 6 * b:9 + 6 * b:2] = np.cos(math.pi * x * 2.0 ** b)
    f[:, 75:78], f[:, 78:81], f[:, 81] = n, wo, 1.0
    pb = np.maximum((wi * n).sum(1), 0.01) / math.pi
    w = np.exp(rng.normal(-0.5, 1.0, rows))
    return f, wi.astype(np.float32), pb.astype(np.float32), w.astype(np.float32), n.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rays", "rays_host"):
        verts, nodes, order = _soup(case["tris"], case["leaf"], case["seed0"])
        rays, n = _rays(case["rays"], case["any"], seed), case["rays"]
        state = {"case": case, "accel": trace.Accel(nodes, order, verts)}
        if kind == "rays":
            state["rays"] = rays
            state["prim"] = torch.empty(n, dtype=torch.int32, device="cuda")
            state["t"] = None if case["any"] else torch.empty(n, dtype=torch.float32, device="cuda")
        else:
            host = torch.empty((n, 8), pin_memory=True)
            host.copy_(rays)
            state["rays"] = host.numpy().reshape(-1).view(abi.RAY)
            state["prim"] = torch.empty(n, dtype=torch.int32).pin_memory().numpy()
            state["t"] = None if case["any"] else torch.empty(n, dtype=torch.float32).pin_memory().numpy()
            state["keep"] = host
        return state
    state = {"case": case, "seed": seed}
    if kind == "v4":
        state["scene"], state["ext"] = _box(case["seed0"], case["w"], case["h"], False, False, False)
    elif kind == "scene_edit":
        state["scene"] = hostscene.build_box_scene(scenes.box_scene(seed=seed, width=case["w"], height=case["h"]))
        state["scene"].desc()
    elif kind == "render":
        state["scene"], state["ext"] = _box(case["seed0"], case["w"], case["h"], case["medium"], case["slit"],
                                            case["light_bvh"])
    elif kind == "outdoor":
        state["scene"], state["ext"] = _outdoor(case["w"], case["h"], case["terrain"], case["cloud"], case["spheres"])
    elif kind == "guided":
        state["scene"], _ = _box(case["seed0"], case["w"], case["h"], False, True, False)
        state["ext"] = render.make_ext(guide=render.GUIDE_SAMPLE)
        guide.set_options()
        guide.set_weights(_guide_weights())
    elif kind == "batch":
        state["renders"] = _batch(case["first"], case["count"], case["div"])
        state["config"] = render.batch_config(1 << 21, 256)
    else:
        state["rows"] = _train_rows(case["rows"], seed)
        guide.set_options()
        guide.set_weights(_guide_weights())
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rays":
        stream = torch.cuda.current_stream().cuda_stream
        t = state["t"]
        state["accel"].trace_device(state["rays"].data_ptr(), case["rays"], state["prim"].data_ptr(),
                                    None if t is None else t.data_ptr(), case["any"], stream)
        return {"prim": state["prim"]} if t is None else {"prim": state["prim"], "t": t}
    if kind == "rays_host":
        state["accel"].trace_host(state["rays"], state["prim"], state["t"], case["any"])
        return {"prim": state["prim"]} if case["any"] else {"prim": state["prim"], "t": state["t"]}
    if kind == "v4":
        return render.render_v4(state["scene"], case["w"], case["h"], case["spp"], seed=state["seed"],
                                max_depth=case["depth"])
    if kind in ("render", "outdoor", "guided"):
        return render.render_ex(state["scene"], case["w"], case["h"], case["spp"], seed=state["seed"],
                                max_depth=case["depth"], ext=state["ext"])
    if kind == "scene_edit":
        return render.render_ex(state["scene"], case["w"], case["h"], case["spp"], seed=state["seed"],
                                max_depth=case["depth"])
    if kind == "batch":
        items = [(hs, None, dict(spp=spp, seed=state["seed"], max_depth=depth), np.zeros((h, w, 3)))
                 for hs, spp, depth, h, w in state["renders"]]
        render.render_batch(items, config=state["config"])
        return [film for _, _, _, film in items]
    f, wi, pb, w, n = state["rows"]
    loss, grad = guide.gradient(f, wi, pb, w, n)
    return {"loss": np.float64(loss), "grad": grad}


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without

# Per ray: the box tests (15 operations each) and triangle tests (40 each) of a binary BVH walk of
# the benchmark soup as the repository's benchmark counts them (28.86 and 2.92 a ray).
_RAY_FLOPS = 28.86 * 15 + 2.92 * 40
# Per path vertex of shading: BSDF, light sampling, spectra at 4 wavelengths.
_VERTEX_FLOPS = 500
_PARAMS = 23552


def _render_work(pixels, spp, depth, prims, vertices):
    """`vertices`: mean closest-hit rays of a path (4.3 in the box at depth 8, more with media);
    two thirds as many shadow rays. Bytes: the film in and out, every primitive once."""
    v = min(vertices, depth + 1)
    return {"bytes": 48 * pixels + 164 * prims, "flops": pixels * spp * v * (_RAY_FLOPS * 5 / 3 + _VERTEX_FLOPS)}


def work(case):
    kind = case["kind"]
    if kind in ("rays", "rays_host"):
        n = case["rays"]
        return {"bytes": n * (36 if case["any"] else 40) + 36 * case["tris"], "flops": n * _RAY_FLOPS}
    if kind == "train":
        # Per row: 128 features, 8 loss inputs, three products per weight (forward, backward, weight gradient).
        return {"bytes": case["rows"] * 4 * 136 + 2 * 4 * _PARAMS, "flops": 6.0 * _PARAMS * case["rows"]}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for s in scenes.uneven_batch(48)[case["first"]:case["first"] + case["count"]]:
            one = _render_work(s.width * s.height, max(1, s.spp // case["div"]), s.max_depth, 44814, 5)
            total = {k: total[k] + one[k] for k in total}
        return total
    prims = 2 * (case["terrain"] - 1) ** 2 + case["spheres"] if kind == "outdoor" else 44814
    one = _render_work(case["w"] * case["h"], case["spp"], case["depth"], prims, 2.5 if kind == "outdoor" else 5)
    if kind == "guided":
        one["flops"] += case["w"] * case["h"] * case["spp"] * 2 * 2.0 * _PARAMS
    return one


def tolerance(case):
    if case["kind"] in ("rays", "rays_host"):
        # Primitive ids and distances are the reference's own bits; only among hits at exactly equal
        # distance may another tree name another primitive.
        return {"rel": 1e-6, "max": 1e-5, "differ": 1e-6}
    if case["kind"] == "train":
        # FP16 activations and signals, FP32 sums: the gradient is 0.0025 (64k rows) to 0.014 (a few
        # thousand) off the one in doubles; sums in another order move it by 1e-7, an activation that
        # rounds to the other FP16 neighbour by about 1e-4.
        return {"rel": 1e-3, "max": 0.02}
    # Films are sums of per-path values in a fixed order, so a render is the same bits each time, and
    # also over a BVH with other leaf sizes (measured: no difference in any listed render). What may
    # move is a path that meets two surfaces at exactly the same distance.
    return {"rel": 1e-3, "max": 0.9}


# ---------------------------------------------------------------------------------------------
# The same in 64 bits


def _exact_rays(case, seed):
    """Brute force: every ray against every triangle (Moller and Trumbore 1997)."""
    if case["any"] or case["rays"] * case["tris"] > 2e10:
        return None
    rays = _rays(case["rays"], case["any"], seed).double()
    v = torch.from_numpy(_soup(case["tris"], case["leaf"], case["seed0"])[0].astype(np.float64)).cuda()
    p0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    best = torch.zeros(case["rays"], dtype=torch.float64, device="cuda")
    step = max(1, int(1.5e8) // case["tris"])
    for i in range(0, case["rays"], step):
        o, d, tmax = rays[i:i + step, None, 0:3], rays[i:i + step, None, 4:7], rays[i:i + step, None, 3]
        p = torch.linalg.cross(d.expand(-1, len(v), 3), e2.expand(len(o), -1, 3))
        inv = 1.0 / (p * e1).sum(-1)
        s = o - p0
        u = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1.expand(len(o), -1, 3))
        w = (d * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        hit = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & (t < tmax)
        t = torch.where(hit, t, math.inf).amin(1)
        best[i:i + step] = torch.where(torch.isinf(t), 0.0, t)
    return {"prim": None, "t": best}


def _exact_train(case, seed):
    """Forward, loss and gradient by automatic differentiation in doubles, nothing rounded to FP16."""
    f, wi, pb, w, n = (torch.from_numpy(a).double().cuda() for a in _train_rows(case["rows"], seed))
    p = torch.from_numpy(_guide_weights()).double().cuda().requires_grad_(True)
    a, at = f, 0
    for k, (rows, cols) in enumerate(((64, 128), (64, 64), (64, 64), (64, 64), (48, 64))):
        z = a @ p[at:at + rows * cols].view(rows, cols).T
        at += rows * cols
        a = z if k == 4 else torch.cat([torch.relu(z[:, :63]), torch.ones_like(z[:, 63:])], 1)
    lobes = a[:, :40].view(-1, 8, 5)
    mu = lobes[..., 0:3] / lobes[..., 0:3].norm(dim=-1, keepdim=True)
    kappa = torch.exp(torch.clamp(lobes[..., 3], -4.0, 8.0))
    pi = torch.softmax(lobes[..., 4], -1)
    mirror = wi - 2.0 * (wi * n).sum(-1, keepdim=True) * n
    norm = kappa / (2.0 * math.pi * -torch.expm1(-2.0 * kappa))
    q = sum((pi * norm * torch.exp(kappa * ((mu * d[:, None]).sum(-1) - 1.0))).sum(-1) for d in (wi, mirror))
    c = 0.5 * torch.sigmoid(a[:, 40])
    loss = -(w * torch.log(q)).sum() - (w * torch.log(c * q.detach() + (1.0 - c) * pb)).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": p.grad}


def exact(case, seed):
    """None for the renders: a path's value hangs on thousands of roundings and decisions, so 64 bits
    trace other paths and give the same image only in expectation."""
    if case["kind"] == "rays":
        return _exact_rays(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
