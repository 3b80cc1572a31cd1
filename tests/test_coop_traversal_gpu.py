"""GPU: the 4-wide ray queries, whose warps finish a launch's last rays together, against the
reference-order binary traversal (prgpu_trace_rays) on the same tree. Sizes lie around one ray a
warp, eight rays a warp and full warps; trees around the depth up to which rays are finished
together (one lane a ray beyond it); leaves shorter and longer than the four lanes of a group."""

import numpy as np
import pytest
import torch

from prgpu import abi, trace, workloads

pytestmark = pytest.mark.gpu


def _tree(leaves):
    """A chain: leaf 0, then the rest, each interior node's first child a leaf of the given triangles."""
    n = len(leaves)
    nodes = np.zeros(2 * n - 1, abi.BVH_NODE)
    for k, (lo, hi, first, count) in enumerate(leaves):
        i = 2 * k + 1 if k < n - 1 else 2 * k
        nodes[i]["bmin"], nodes[i]["bmax"], nodes[i]["offset"], nodes[i]["nPrims"] = lo, hi, first, count
        if k < n - 1:
            rest = leaves[k:]
            nodes[2 * k]["bmin"] = np.min([x[0] for x in rest], axis=0)
            nodes[2 * k]["bmax"] = np.max([x[1] for x in rest], axis=0)
            nodes[2 * k]["offset"] = 2 * k + 2
    return nodes


def _chain(levels, per_leaf, seed):
    """`levels` leaves of `per_leaf` soup triangles each, in a chain of interior nodes."""
    verts = workloads.triangle_soup(levels * per_leaf, seed=seed, edge=0.3)
    boxes = [(verts[k * per_leaf:(k + 1) * per_leaf].min((0, 1)), verts[k * per_leaf:(k + 1) * per_leaf].max((0, 1)),
              k * per_leaf, per_leaf) for k in range(levels)]
    return verts, _tree(boxes), np.arange(levels * per_leaf, dtype=np.int32)


def _check(nodes, order, verts, rays, any_hit):
    want = trace.trace_rays(nodes, order, verts, rays, any_hit=any_hit)
    accel = trace.Accel(nodes, order, verts)
    n = len(rays)
    dev = torch.from_numpy(np.ascontiguousarray(rays).view(np.float32).reshape(n, 8).copy()).cuda()
    prim = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    t = torch.full((n,), -7.0, device="cuda")
    accel.trace_device(dev.data_ptr(), n, prim.data_ptr(), None if any_hit else t.data_ptr(), any_hit,
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert accel.status() == 0
    prim, t = prim.cpu().numpy(), t.cpu().numpy()
    if any_hit:
        np.testing.assert_array_equal(prim, want)
        return want
    np.testing.assert_array_equal(t.view(np.int32), want[1].view(np.int32))
    np.testing.assert_array_equal(prim >= 0, want[0] >= 0)
    # Another primitive only where each of the two, alone, is hit at exactly that distance.
    for k in np.flatnonzero(prim != want[0]):
        for p in (prim[k], want[0][k]):
            v = verts[p:p + 1]
            one = _tree([(v.min((0, 1)), v.max((0, 1)), 0, 1)])
            alone = trace.trace_rays(one, np.zeros(1, np.int32), v, rays[k:k + 1])
            assert alone[0][0] == 0 and alone[1].view(np.int32)[0] == t.view(np.int32)[k]
    return want[0]


def _rays(n, any_hit, seed):
    rays = workloads.soup_rays(n, seed=seed, any_hit=any_hit)
    rays["d"][::7, seed % 3] = 0.0  # directions with infinite reciprocals
    rays["d"][3::11, :2] = 0.0
    rays["tMax"][::13] = 0.25
    return rays


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("n", [1, 7, 33, 1000, 4735, 4737, 37888, 37897, 151553, 400009, (3 << 20) + 5])
def test_sizes(gpu, n, any_hit):
    verts = workloads.triangle_soup(20011, seed=3, edge=0.04)
    nodes, order = trace.build_bvh_triangles(verts, max_leaf=4)
    got = _check(nodes, order, verts, _rays(n, any_hit, 5), any_hit)
    if n >= 1000:
        assert 0 < (got > 0).sum() < n


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("levels,per_leaf", [(1, 1), (1, 3), (1, 11), (2, 4), (5, 5), (30, 2), (38, 1), (41, 3), (60, 2)])
def test_leaves_and_depths(gpu, levels, per_leaf, any_hit):
    verts, nodes, order = _chain(levels, per_leaf, levels)
    for n in (40, 20000):
        _check(nodes, order, verts, _rays(n, any_hit, 2), any_hit)


def test_distance_that_is_not_a_number(gpu):
    """Triangles so small that the reciprocal of the determinant overflows are hit at a distance that
    is not a number, after which the visit order decides: one leaf, whose order both forms share."""
    verts = np.zeros((3, 3, 3), np.float32)
    verts[:, 1, 0] = verts[:, 2, 1] = [0.75, 1e-20, 3e-20]
    verts[0, 0, :2] = verts[0, 1, 1] = verts[0, 2, 0] = -0.25
    verts[0, :, 2] = 0.25
    nodes = _tree([(verts.min((0, 1)), verts.max((0, 1)), 0, 3)])
    rays = workloads.soup_rays(70, seed=1)
    rays["o"] = [0.0, 0.0, -1e-10]  # the numerator underflows to 0, its product with infinity is no number
    rays["d"] = [0.0, 0.0, 1.0]
    rays["o"][::2, :2] = 0.125
    want = trace.trace_rays(nodes, np.arange(3, dtype=np.int32), verts, rays)
    assert np.isnan(want[1]).any() and (want[1] == 0.25).any()
    _check(nodes, np.arange(3, dtype=np.int32), verts, rays, False)
