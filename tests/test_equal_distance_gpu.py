"""GPU: surfaces that lie on one another. Which of several hits at the same distance wins hangs on the
order in which the leaves are visited, so that order must be the ray's own (depth first, nearest child
first) and not the schedule's: the same whether a ray was traced by one lane to its end or finished by
its whole warp, and so the same in every run, for every queue length and in every batch.

The one-lane results to compare with come from queries long enough for the kernel without the
cooperative tail, and for renders from the same scene under a chain of far-away triangles, whose tree is
too deep for it (the scene's own part of the tree is unchanged)."""

import numpy as np
import pytest
import torch

from prgpu import abi, hostscene, render, scenes, spectra, trace, workloads

pytestmark = pytest.mark.gpu

LONG = (3 << 20) + 1  # rays from which a query takes the kernel without the cooperative tail


def _device_trace(accel, rays):
    n = len(rays)
    dev = torch.from_numpy(np.ascontiguousarray(rays).view(np.float32).reshape(n, 8).copy()).cuda()
    prim = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    t = torch.full((n,), -7.0, device="cuda")
    accel.trace_device(dev.data_ptr(), n, prim.data_ptr(), t.data_ptr(), False, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert accel.status() == 0
    return prim.cpu().numpy(), t.cpu().numpy()


def _copies(verts, k, seed):
    """Every triangle k times, in shuffled order."""
    v = np.repeat(verts, k, axis=0)
    return np.ascontiguousarray(v[np.random.default_rng(seed).permutation(len(v))])


def _tiles(n, seed):
    """Axis-aligned right triangles on a few common planes: flat boxes, entered at about the distance of
    the hit, on either side of it by rounding."""
    rng = np.random.default_rng(seed)
    axis = rng.integers(0, 3, n)
    c = rng.random((n, 3)).astype(np.float32)
    c[np.arange(n), axis] = np.float32(0.1) + np.float32(0.13) * rng.integers(0, 6, n).astype(np.float32)
    v = np.repeat(c[:, None, :], 3, axis=1)
    v[np.arange(n), 1, (axis + 1) % 3] += rng.uniform(0.05, 0.3, n).astype(np.float32)
    v[np.arange(n), 2, (axis + 2) % 3] += rng.uniform(0.05, 0.3, n).astype(np.float32)
    return v


def _ulp(verts, seed):
    """Copies whose corners differ by one unit in the last place: distances that nearly tie."""
    rng = np.random.default_rng(seed)
    up = np.nextafter(verts, np.float32(4.0))
    return np.concatenate([verts, np.where(rng.random(verts.shape) < 0.5, up, verts)])


GEOMETRY = {
    "soup": lambda: _copies(workloads.triangle_soup(1500, seed=1, edge=0.15), 4, 1),
    "tiles": lambda: _copies(_tiles(700, 2), 3, 2),
    "ulp": lambda: _copies(_ulp(_tiles(900, 3), 4), 2, 3),
    "stack": lambda: _copies(workloads.triangle_soup(40, seed=5, edge=0.6), 30, 5),
}


@pytest.mark.parametrize("max_leaf", [1, 4])
@pytest.mark.parametrize("kind", sorted(GEOMETRY))
def test_queries_do_not_depend_on_the_schedule(gpu, kind, max_leaf):
    verts = GEOMETRY[kind]()
    nodes, order = trace.build_bvh_triangles(verts, max_leaf=max_leaf)
    accel = trace.Accel(nodes, order, verts)
    rays = workloads.soup_rays(60000, seed=7)
    rays["d"][::9, 1] = 0.0
    prim, t = _device_trace(accel, np.resize(rays, LONG))
    np.testing.assert_array_equal(prim[:3000], prim[60000:63000])
    assert (prim[:60000] >= 0).mean() > 0.2
    for n in (1, 500, 4736, 20000, 60000):
        for _ in range(3):
            got, gt = _device_trace(accel, rays[:n])
            np.testing.assert_array_equal(gt.view(np.int32), t[:n].view(np.int32))
            np.testing.assert_array_equal(got, prim[:n])


def test_boxes_that_stick_out_of_their_parents(gpu):
    """The caller's boxes need not be nested; a child entered before its parent is then visited or not as
    the one-lane walk's tMax at the parent has it."""
    verts = GEOMETRY["ulp"]()
    nodes, order = trace.build_bvh_triangles(verts, max_leaf=2)
    rng = np.random.default_rng(8)
    inner = np.flatnonzero(nodes["nPrims"] == 0)[1:]
    inner = inner[rng.random(len(inner)) < 0.3]
    low, high = nodes["bmin"][inner].copy(), nodes["bmax"][inner].copy()
    f = rng.uniform(0.0, 0.25, (2, len(inner), 3)).astype(np.float32)
    nodes["bmin"][inner], nodes["bmax"][inner] = low + f[0] * (high - low), high - f[1] * (high - low)
    accel = trace.Accel(nodes, order, verts)
    rays = workloads.soup_rays(20000, seed=9)
    prim, t = _device_trace(accel, np.resize(rays, LONG))
    for n in (300, 20000):
        got, gt = _device_trace(accel, rays[:n])
        np.testing.assert_array_equal(gt.view(np.int32), t[:n].view(np.int32))
        np.testing.assert_array_equal(got, prim[:n])


def test_a_distance_that_is_not_a_number_among_many_leaves(gpu):
    """A triangle so small that its reciprocal determinant overflows is hit at a distance that is not a
    number, after which nothing is nearer: whatever the one-lane walk meets first decides. Leaves of one
    plain triangle, every third with such a one before or after it, under a balanced tree."""
    rng = np.random.default_rng(3)
    tiny = np.zeros((3, 3), np.float32)
    tiny[1, 0] = tiny[2, 1] = 1e-20
    verts, leaves = [], []
    for k in range(48):
        plain = rng.uniform(-0.4, 0.4, (3, 3)).astype(np.float32)
        plain[:, 2] = rng.uniform(0.05, 0.6)
        own = [plain] if k % 3 else ([tiny, plain] if k % 2 else [plain, tiny])
        low, high = np.array([-0.5, -0.5, rng.uniform(-0.1, 0.04)]), np.array([0.5, 0.5, 0.7])
        leaves.append((low, high, len(verts), len(own)))
        verts += own
    nodes = np.zeros(2 * len(leaves) - 1, abi.BVH_NODE)

    def build(lo, hi, at):
        n = nodes[at]
        n["bmin"] = np.min([x[0] for x in leaves[lo:hi]], axis=0)
        n["bmax"] = np.max([x[1] for x in leaves[lo:hi]], axis=0)
        if hi - lo == 1:
            n["offset"], n["nPrims"] = leaves[lo][2:]
            return at + 1
        mid = (lo + hi) // 2
        n["offset"] = build(lo, mid, at + 1)
        return build(mid, hi, int(n["offset"]))

    assert build(0, len(leaves), 0) == len(nodes)
    accel = trace.Accel(nodes, np.arange(len(verts), dtype=np.int32), np.array(verts))
    rays = workloads.soup_rays(300, seed=1)
    rays["o"] = [0.0, 0.0, -1e-10]  # the numerator underflows to 0, its product with infinity is no number
    rays["d"] = [0.0, 0.0, 1.0]
    rays["o"][1::2, :2] = rng.uniform(-0.2, 0.2, (150, 2))
    rays["tMax"][::5] = rng.uniform(1e-3, 0.3, 60)
    prim, t = _device_trace(accel, np.resize(rays, LONG))
    assert np.isnan(t[:300]).sum() > 50 and (t[:300] > 0.0).sum() > 50
    for n in (1, 2, 7, 300):
        got, gt = _device_trace(accel, rays[:n])
        np.testing.assert_array_equal(gt.view(np.int32), t[:n].view(np.int32))
        np.testing.assert_array_equal(got, prim[:n])


# ---------------------------------------------------------------------------------------------
# Renders


def _scene(spheres=False, walls=False, fog=False, seed=0):
    """A small lit room in which every surface lies on another of a different colour; with analytic
    spheres (two materials on each), and with a medium inside interface walls."""
    s = scenes.box_scene(seed=seed, width=40, height=36, subdiv=1)
    s.spheres = s.spheres[:12]
    h = hostscene.HostScene()
    rng = np.random.default_rng(seed)
    mats = [h.material(type=abi.MAT_DIFFUSE, albedo=h.spectrum(spectra.constant(float(a)))) for a in (0.1, 0.8, 0.4, 0.6)]
    light = h.spectrum(spectra.blackbody(6500.0))
    inside = h.medium(spectra.constant(0.2), spectra.constant(0.6), 0.3) if walls or fog else -1
    if fog:
        h.camera_medium = inside
    out = inside if fog else -1
    for _, _, quad in scenes.wall_quads():
        for k in rng.permutation(4)[:3]:
            h.mesh(np.asarray(quad, np.float32), [0, 1, 2, 0, 2, 3], mats[k], medium_inside=out, medium_outside=out)
    h.mesh(np.asarray([[-0.5, 0.999, -0.5], [0.5, 0.999, -0.5], [0.5, 0.999, 0.5], [-0.5, 0.999, 0.5]], np.float32),
           [0, 1, 2, 0, 2, 3], mats[0], normals=np.tile([0.0, -1.0, 0.0], (4, 1)),
           light_spectrum=light, light_scale=30.0, medium_inside=out, medium_outside=out)
    for sp in s.spheres:
        p, n, f = scenes.sphere_mesh(sp, 1)
        for k in rng.permutation(4)[:2]:
            h.mesh(p, f, mats[k], normals=n, medium_inside=out, medium_outside=out)
    if spheres:
        c = rng.uniform(-0.6, 0.6, (25, 3))
        r = rng.uniform(0.05, 0.2, 25)
        for k in (0, 1, 3):
            h.spheres(c, r, rng.permutation(np.resize([mats[k], mats[2]], 25)), medium_inside=out, medium_outside=out)
    if walls:
        v, f = hostscene.box_mesh([-0.7, -0.6, -0.6], [0.7, 0.3, 0.5])
        h.mesh(v, f, h.material(type=abi.MAT_INTERFACE), medium_inside=inside, medium_outside=-1)
        h.mesh(v[:, [1, 2, 0]] * 0.5, f, h.material(type=abi.MAT_INTERFACE), medium_inside=inside, medium_outside=inside)
    return h.finish(cam_pos=(0.0, -0.1, 0.95), cam_target=(0.0, -0.2, -0.3), fov_y=65.0, width=40, height=36)


def _deep(h, levels=45):
    """The same scene under a chain of `levels` far-away triangles: too deep a tree for the cooperative
    tail. A multiple of three, so that the scene's own root is again the root of a 4-wide node."""
    n = len(h.prim_array)
    extra = np.zeros(levels, abi.PRIMITIVE)
    extra["type"], extra["material"], extra["light"] = abi.PRIM_TRIANGLE, 0, -1
    extra["mediumInside"] = extra["mediumOutside"] = h.camera_medium
    at = np.stack([300.0 + np.arange(levels), np.full(levels, 300.0), np.full(levels, 300.0)], 1).astype(np.float32)
    extra["p0"], extra["p1"], extra["p2"] = at, at + [0.1, 0, 0], at + [0, 0.1, 0]
    nodes = np.zeros(2 * levels + len(h.nodes), abi.BVH_NODE)
    low, high = h.nodes[0]["bmin"], h.nodes[0]["bmax"]
    for k in range(levels):
        leaf = nodes[2 * k + 1]
        leaf["bmin"], leaf["bmax"], leaf["offset"], leaf["nPrims"] = at[k], at[k] + [0.1, 0.1, 0.0], n + k, 1
        nodes[2 * k]["bmin"], nodes[2 * k]["bmax"] = np.minimum(low, at[k]), np.maximum(high, at[-1] + 0.1)
        nodes[2 * k]["offset"] = 2 * k + 2
    own = nodes[2 * levels:]
    own[:] = h.nodes
    own["offset"][own["nPrims"] == 0] += 2 * levels
    h.prim_array = np.concatenate([h.prim_array, extra])
    h.nodes, h.order = nodes, np.concatenate([h.order, np.arange(n, n + levels, dtype=np.int32)])
    h._desc = None
    return h


VARIANTS = {"plain": {}, "fog": {"fog": True}, "spheres": {"spheres": True}, "walls": {"walls": True},
            "spheres_walls": {"spheres": True, "walls": True}, "spheres_fog": {"spheres": True, "fog": True}}


def _render(h, paths):
    ext = render.make_ext(wavefront_paths=paths)
    return render.render_ex(h, 40, 36, 6, seed=11, max_depth=7, ext=ext)


@pytest.mark.parametrize("variant", sorted(VARIANTS))
def test_films_do_not_depend_on_the_schedule(gpu, variant):
    want = _render(_deep(_scene(**VARIANTS[variant])), 1 << 20)
    assert np.isfinite(want).all() and want[..., 1].mean() > 0
    h = _scene(**VARIANTS[variant])
    for paths in (1 << 20, 2000, 1024):
        for _ in range(2):
            np.testing.assert_array_equal(_render(h, paths), want)


@pytest.mark.parametrize("variants", [("plain", "spheres"), ("plain", "fog"), ("walls", "spheres_walls"),
                                      ("plain", "walls"), ("spheres_fog", "fog")])
def test_batches_of_shallow_and_deep_trees(gpu, variants):
    """Rays of several scenes in one warp, each against its own tree, with trees on both sides of the
    depth up to which rays are finished together."""
    scenes_ = [f(_scene(**VARIANTS[v], seed=k)) for k, v in enumerate(variants) for f in (lambda x: x, _deep)]
    films = [np.zeros((36, 40, 3)) for _ in scenes_]
    render.render_batch([(h, None, dict(spp=6, seed=11, max_depth=7), film) for h, film in zip(scenes_, films)],
                        config=render.batch_config(1 << 14, 256))
    for k in range(0, len(scenes_), 2):
        one = _render(scenes_[k + 1], 1 << 20)
        np.testing.assert_array_equal(films[k + 1], one)
        np.testing.assert_array_equal(films[k], one)
