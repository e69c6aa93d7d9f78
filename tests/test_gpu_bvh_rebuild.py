"""Device rebuilds (tfgTinyBVHConstruirGPU) at the sizes where the eight-lane
collapse and the single result allocation change: leaf and node counts around
8 children, gaps among the triangles that break the warp copies, trees deeper
than one batch of levels, trees with more nodes than the result block has room
for, and rebuilds on several streams at once."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tfg_b200 import _lib
from tfg_b200 import bvh as hbvh
from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes
from tfg_b200.devmem import view_device
from tfg_b200.structs import PRIMITIVA, TRIANGULO, CTinyBVH

pytestmark = pytest.mark.gpu


def _mesh(tris):
    m = np.zeros(len(tris), PRIMITIVA)
    m["tipo"] = TRIANGULO
    m["u"][:, :9] = np.asarray(tris, np.float64).reshape(len(tris), 9)
    return m


def _cloud(n, seed, size=0.2):
    rng = np.random.default_rng(seed)
    return (rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(size=(n, 3, 3)) * size).reshape(n, 9)


def _growing(n, ratio, seed, spread):
    """Triangles whose distance from the origin grows geometrically: deep, thin trees."""
    rng = np.random.default_rng(seed)
    c = (ratio ** np.arange(n))[:, None, None]
    return (c * np.ones((1, 3, 3)) + rng.normal(size=(n, 3, 3)) * spread * c).reshape(n, 9)


def _build(mesh, stream=0):
    d = torch.from_numpy(mesh.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    b = CTinyBVH()
    _lib.call("tfgTinyBVHConstruirGPU", d.data_ptr(), len(mesh), ctypes.byref(b), stream)
    return b


def _trace(b, rays):
    dr = torch.from_numpy(rays.reshape(-1).copy()).cuda()
    hits = torch.zeros(len(rays) * 4, device="cuda")
    _lib.call("tfgTraceRays", ctypes.byref(b.ref), b.d_tris_wt, pt.TRIS_REF, dr.data_ptr(), len(rays),
              hits.data_ptr(), 0)
    torch.cuda.synchronize()
    return hits.view(-1, 4).cpu().numpy()


def _rays_at(tris, n, seed):
    """Rays toward points of the triangles."""
    rng = np.random.default_rng(seed)
    t = np.asarray(tris, np.float64).reshape(-1, 3, 3)[rng.integers(0, len(tris), n)]
    w = rng.dirichlet((1, 1, 1), n)
    target = (t * w[:, :, None]).sum(1)
    o = target + rng.normal(size=(n, 3)) * (np.abs(target).max(1, keepdims=True) + 0.5)
    d = target - o
    r = np.zeros((n, 8), np.float32)
    r[:, :3], r[:, 4:7], r[:, 3] = o, d / np.linalg.norm(d, axis=1, keepdims=True), 1e9
    return r


def _check(b, mesh, tris, seed):
    nt = len(tris)
    assert b.ref.num_tris == nt and b.num_primitivas == nt
    prims = view_device(b.d_primitivas, nt * PRIMITIVA.itemsize, np.uint8).cpu().numpy()
    np.testing.assert_array_equal(prims, np.ascontiguousarray(mesh[mesh["tipo"] == TRIANGULO]).view(np.uint8))
    ids = view_device(b.d_tris_wt, nt * 12).cpu().numpy().reshape(nt, 12)[:, 3].view(np.uint32)
    assert sorted(ids.tolist()) == list(range(nt))
    hb = hbvh.build_host(hbvh.triangle_vertices(mesh))
    rays = _rays_at(tris, 2000, seed)
    got, want = _trace(b, rays), orc.brute_batch(hb.tris_ref, rays)
    np.testing.assert_array_equal(got[:, 3].view(np.uint32), want[:, 3].view(np.uint32))


@pytest.mark.parametrize("n", [3, 4, 7, 8, 9, 24, 25, 33, 257, 1000])
def test_rebuild_hits_equal_brute_force(built, n):
    tris = _cloud(n, n)
    b = _build(_mesh(tris))
    _check(b, _mesh(tris), tris, n)
    _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))


@pytest.mark.parametrize("gap", [1, 31, 32, 33])
def test_triangles_between_other_primitives(built, gap):
    tris = _cloud(150, gap)
    mesh = _mesh(tris)
    sphere = scenes.sphere_prim((0.0, 0.0, 30.0), 0.5)
    mesh = np.concatenate([x for k in range(0, 150, gap) for x in (mesh[k:k + gap], sphere)])
    b = _build(mesh)
    _check(b, mesh, tris, gap)
    _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))


@pytest.mark.parametrize("n,ratio,spread,deep,own_nodes", [(2000, 1.01, 1.0, True, False),
                                                           (1500, 1.02, 0.01, True, True)])
def test_deep_and_node_rich_trees(built, n, ratio, spread, deep, own_nodes):
    tris = _growing(n, ratio, 3, spread)
    mesh = _mesh(tris)
    b = _build(mesh)
    assert (b.max_depth > 8) == deep
    assert (b.ref.num_nodos > n // 8 + 16) == own_nodes
    ids = view_device(b.d_tris_wt, n * 12).cpu().numpy().reshape(n, 12)[:, 3].view(np.uint32)
    assert sorted(ids.tolist()) == list(range(n))
    hb = hbvh.build_host(hbvh.triangle_vertices(mesh))
    rays = _rays_at(tris, 2000, 9)
    got, want = _trace(b, rays), orc.brute_batch(hb.tris_ref, rays)
    assert (got[:, 3].view(np.uint32) != want[:, 3].view(np.uint32)).mean() < 5e-3   # equal-t ties
    _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))


def test_rebuilds_on_several_streams_at_once(built):
    clouds = [_cloud(n, n) for n in (500, 2000, 7000)]
    want = []
    for t in clouds:
        b = _build(_mesh(t))
        want.append(_trace(b, _rays_at(t, 500, 1)))
        _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))
    bad = []

    def work(k):
        s = torch.cuda.Stream()
        for _ in range(10):
            b = _build(_mesh(clouds[k]), s.cuda_stream)
            if not np.array_equal(_trace(b, _rays_at(clouds[k], 500, 1)), want[k], equal_nan=True):
                bad.append(k)
            _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
