"""GPU: one ray-query handle used from several streams and threads at a time, from host buffers at the
same time, and captured in CUDA graphs. Every query draws its rays from a counter; each must get all of
its own rays, each once, whatever else is in flight."""

import ctypes as C
import threading

import numpy as np
import pytest
import torch

from prgpu import trace, workloads

pytestmark = pytest.mark.gpu

SIZES = (777, 40001, 300007, 90000, 1500001, 5)


@pytest.fixture(scope="module")
def scene(gpu):
    verts = workloads.triangle_soup(60000, seed=2, edge=0.03)
    nodes, order = trace.build_bvh_triangles(verts)
    accel = trace.Accel(nodes, order, verts)
    rays = workloads.soup_rays(max(SIZES), seed=4)
    dev = torch.from_numpy(np.ascontiguousarray(rays).view(np.float32).reshape(-1, 8).copy()).cuda()
    prim, t = (x.cpu().numpy() for x in _launch(accel, dev, max(SIZES), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert accel.status() == 0 and 0.2 < (prim >= 0).mean() < 1.0
    return accel, rays, dev, prim, t


def _out(n):
    return torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.full((n,), -7.0, device="cuda")


def _launch(accel, dev, n, stream, out=None):
    prim, t = out or _out(n)
    accel.trace_device(dev.data_ptr(), n, prim.data_ptr(), t.data_ptr(), False, stream)
    return prim, t


def _same(got, want_prim, want_t):
    n = len(got[0])
    np.testing.assert_array_equal(got[0].cpu().numpy(), want_prim[:n])
    np.testing.assert_array_equal(got[1].cpu().numpy().view(np.int32), want_t[:n].view(np.int32))


def test_streams_at_the_same_time(scene):
    accel, _, dev, prim, t = scene
    streams = [torch.cuda.Stream() for _ in SIZES]
    outs = [[_out(n) for n in SIZES] for _ in range(4)]
    torch.cuda.synchronize()
    for row in outs:
        for s, n, o in zip(streams, SIZES, row):
            _launch(accel, dev, n, s.cuda_stream, o)
    # The status word answers for all of them, without a synchronisation by the caller.
    assert accel.status() == 0
    for row in outs:
        for o in row:
            _same(o, prim, t)


@pytest.mark.parametrize("shared", [False, True])
def test_threads_and_host_queries_at_the_same_time(scene, shared):
    """Threads on their own streams or all on one, while another thread queries from host buffers."""
    accel, rays, dev, prim, t = scene
    one = torch.cuda.Stream()
    bad = []

    def device_queries(k):
        try:
            s = one if shared else torch.cuda.Stream()
            n = SIZES[k % len(SIZES)]
            outs = [_out(n) for _ in range(8)]
            torch.cuda.synchronize()
            for o in outs:
                _launch(accel, dev, n, s.cuda_stream, o)
            s.synchronize()
            for o in outs:
                _same(o, prim, t)
        except BaseException as e:  # noqa: BLE001
            bad.append(e)

    def host_queries():
        try:
            for n in (1200001, 70001):
                p, d = np.full(n, -7, np.int32), np.full(n, -7.0, np.float32)
                accel.trace_host(rays[:n], p, d, False)
                np.testing.assert_array_equal(p, prim[:n])
                np.testing.assert_array_equal(d.view(np.int32), t[:n].view(np.int32))
        except BaseException as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=device_queries, args=(k,)) for k in range(6)]
    threads.append(threading.Thread(target=host_queries))
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad, bad[0]
    assert accel.status() == 0


def test_captured_queries_beside_others(scene):
    """Two graphs captured on one stream, replayed on two others while that stream goes on."""
    accel, _, dev, prim, t = scene
    outs = [_out(300007), _out(90000)]
    base = torch.cuda.Stream()
    graphs = []
    for o in outs:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=base):
            _launch(accel, dev, len(o[0]), torch.cuda.current_stream().cuda_stream, o)
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(5):
        eager = _out(40001)
        for o in outs:
            o[0].fill_(-7)
            o[1].fill_(-7.0)
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        _launch(accel, dev, 40001, base.cuda_stream, eager)
        torch.cuda.synchronize()
        for o in (*outs, eager):
            _same(o, prim, t)
    assert accel.status() == 0


def test_more_streams_than_counters_are_set_aside(gpu):
    """Streams that come and go, the last of them capturing: the handle's counters are added to meanwhile."""
    verts = workloads.triangle_soup(2000, seed=2, edge=0.05)
    nodes, order = trace.build_bvh_triangles(verts)
    accel = trace.Accel(nodes, order, verts)
    n = 1000
    dev = torch.from_numpy(np.ascontiguousarray(workloads.soup_rays(n, seed=4)).view(np.float32).reshape(n, 8).copy()).cuda()
    want = _launch(accel, dev, n, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    prim, t = want[0].cpu().numpy(), want[1].cpu().numpy()
    cu = C.CDLL("libcuda.so.1")
    for k in range(254):  # with the one above, all that a new handle has
        h = C.c_void_p()
        assert cu.cuStreamCreate(C.byref(h), 1) == 0
        got = _launch(accel, dev, n, h.value)
        assert cu.cuStreamSynchronize(h) == 0
        if k % 50 == 0:
            _same(got, prim, t)
        assert cu.cuStreamDestroy_v2(h) == 0
    out = _out(n)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _launch(accel, dev, n, torch.cuda.current_stream().cuda_stream, out)
    g.replay()
    torch.cuda.synchronize()
    _same(out, prim, t)
    _same(_launch(accel, dev, n, torch.cuda.Stream().cuda_stream), prim, t)
    assert accel.status() == 0
