"""Short queues (eight lanes per ray, k_few) against the one-lane kernels.

The work-counting variants of the traversal stages run every queue with one
lane per ray, so a pass with PROFILE_COUNTS is the reference for the same pass
without it: images, training records and cache queries must be equal bit for
bit -- around one and several rounds of groups, for every number of lights
that changes how a point's shadow rays share a warp, for both triangle
formats, analytic primitives of every kind (also more than eight, and more
than a block caches), no mesh, no lights, wavefronts that start short and
wavefronts whose later bounces become short, and batches."""
import numpy as np
import pytest
import torch

from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes
from tfg_b200.structs import PRIMITIVA

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_tuning():
    pt.set_tuning(pt.RenderTuning.default())
    yield
    pt.set_tuning(pt.RenderTuning.default())


def _pass(ds, counts, depth=8, fmt=pt.TRIS_WATERTIGHT, shadow_mesh=1, frame=5):
    n = ds.scene.width * ds.scene.height
    p = pt.RenderParams(max_depth=depth, rr_min_depth=3, shadow_mesh=shadow_mesh, tri_format=fmt, spp=1, accumulate=1,
                        profile=pt.PROFILE_COUNTS if counts else 0)
    img = torch.zeros(n * 3, device="cuda")
    acc = torch.zeros(n * 3, device="cuda")
    pt.render_pass(ds, p, frame, img, acc)
    torch.cuda.synchronize()
    return img.cpu().numpy(), acc.cpu().numpy()


def _check(ds, **kw):
    got, want = _pass(ds, False, **kw), _pass(ds, True, **kw)
    assert np.isfinite(want[1]).all()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


def _lights(n):
    return scenes.lights(*[((np.cos(2.1 * k), 1.2 + 0.1 * k, 0.8 + np.sin(2.1 * k)), (9.0, 8.0, 7.0 + k))
                           for k in range(n)])


# 1 path; one block's 16 groups and their neighbours; a partly filled last
# warp; 65,536 paths (the largest wavefront k_few runs alone, several rounds)
# and one row more (its later bounces become short)
@pytest.mark.parametrize("w,h", [(1, 1), (4, 4), (17, 1), (33, 31), (256, 256), (256, 257)])
@pytest.mark.parametrize("fmt", [pt.TRIS_REF, pt.TRIS_WATERTIGHT])
def test_short_queues_equal_one_lane_kernels(built, w, h, fmt):
    ds = pt.DeviceScene(scenes.reference_room(w, h, subdiv=2), "cuda")
    _check(ds, fmt=fmt)
    ds.close()


@pytest.mark.parametrize("nl", [0, 1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("shadow_mesh", [0, 1])
def test_lights_of_a_point(built, nl, shadow_mesh):
    s = scenes.tiny_box(61, 47, subdiv=3)
    s.lights = _lights(nl)
    ds = pt.DeviceScene(s, "cuda")
    _check(ds, shadow_mesh=shadow_mesh)
    ds.close()


@pytest.mark.parametrize("nprims", [0, 1, 7, 8, 9, 40, 130])
def test_analytic_primitives(built, nprims):
    base = scenes.reference_room(40, 33, subdiv=1)
    rng = np.random.default_rng(nprims)
    prims = np.concatenate([base.prims, base.prims[:0]] + [
        scenes.sphere_prim(rng.uniform((-3, -2, -6), (3, 2, -1)), float(rng.uniform(0.05, 0.4)), kd=(0.5, 0.4, 0.3))
        for _ in range(max(0, nprims - len(base.prims)))])[:nprims]
    for mesh in (base.mesh, base.mesh[:0]):
        s = scenes.Scene(prims, mesh, base.lights, base.camera, 40, 33, bounds=base.bounds)
        if not len(prims):
            s.prims = np.zeros(0, PRIMITIVA)
        ds = pt.DeviceScene(s, "cuda")
        _check(ds)
        ds.close()


def test_equal_distances_keep_the_first_primitive(built):
    # coincident analytic triangles of different colours, and coincident mesh triangles
    base = scenes.tiny_box(48, 40, subdiv=1)
    prims = np.concatenate([base.prims, base.prims, base.prims])
    for k, c in enumerate(("r", "g", "b")):
        prims["difuso"][c][12 * k:12 * k + 12] = 0.2 + 0.25 * k
    mesh = np.concatenate([base.mesh, base.mesh])
    mesh["difuso"]["r"][len(base.mesh):] = 0.9
    ds = pt.DeviceScene(scenes.Scene(prims, mesh, base.lights, base.camera, 48, 40, bounds=base.bounds), "cuda")
    _check(ds)
    ds.close()


def test_cache_passes_with_short_queues(built):
    ds = pt.DeviceScene(scenes.reference_room(96, 64, subdiv=2), "cuda")
    n = 96 * 64
    outs = []
    for profile in (0, pt.PROFILE_COUNTS):
        nrc = pt.NrcBuffers(n, "cuda")
        img = torch.zeros(n * 3, device="cuda")
        p = pt.RenderParams(max_depth=12, rr_min_depth=5, shadow_mesh=1, profile=profile)
        pt.render_pass(ds, p, 3, img, None, nrc, use_inf=True, train=True)
        torch.cuda.synchronize()
        k = int(nrc.counter.item())
        # records land in the ring in any order
        regs = sorted(bytes(r) for r in nrc.regs.cpu().numpy().reshape(-1, 232)[:k])
        outs.append((img.cpu().numpy(), nrc.infer.cpu().numpy(), nrc.thr.cpu().numpy(), regs))
    for a, b in zip(outs[0][:3], outs[1][:3]):
        np.testing.assert_array_equal(a, b)
    assert outs[0][3] == outs[1][3] and len(outs[0][3]) > 0
    ds.close()


@pytest.mark.parametrize("sizes", [((24, 16), (9, 7), (31, 33)), ((300, 200), (160, 90), (64, 64))])
def test_batches_with_short_queues(built, sizes):
    dss = []
    for k, (w, h) in enumerate(sizes):
        s = scenes.reference_room(w, h, subdiv=2) if k % 2 else scenes.tiny_box(w, h, subdiv=3)
        s.lights = _lights(k + 1)
        dss.append(pt.DeviceScene(s, "cuda"))
    outs = []
    for profile in (0, pt.PROFILE_COUNTS):
        p = pt.RenderParams(max_depth=6, rr_min_depth=3, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=1,
                            accumulate=1, profile=profile)
        accs = [torch.zeros(d.scene.width * d.scene.height * 3, device="cuda") for d in dss]
        pt.render_pass_batch(dss, p, 7, None, accs)
        torch.cuda.synchronize()
        outs.append([a.cpu().numpy() for a in accs])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    for d in dss:
        d.close()


@pytest.mark.parametrize("w,h", [(64, 48), (300, 256)])   # k_few alone; beside the long-queue kernels
def test_passes_that_follow_each_other_closely(built, w, h):
    """Kernels of short wavefronts start before their predecessors end: passes
    back to back, in several wavefronts each, with writes to what they read
    between them, directly and as a replayed graph."""
    ds = pt.DeviceScene(scenes.reference_room(w, h, subdiv=2), "cuda")
    n = w * h
    p = pt.RenderParams(max_depth=6, rr_min_depth=3, shadow_mesh=1, spp=2, accumulate=1)
    imgs = [torch.zeros(n * 3, device="cuda") for _ in range(4)]
    acc = torch.zeros(n * 3, device="cuda")

    def passes():
        acc.zero_()
        for k, img in enumerate(imgs):
            pt.render_pass(ds, p, 2 * k, img, acc)
            acc.mul_(0.5)

    want = []
    for k in range(4):   # one at a time
        if k == 0:
            acc.zero_()
        pt.render_pass(ds, p, 2 * k, imgs[k], acc)
        torch.cuda.synchronize()
        acc.mul_(0.5)
        torch.cuda.synchronize()
    want = [acc.clone()] + [i.clone() for i in imgs]

    for wavefront in (0, n // 3):
        pt.set_tuning(pt.RenderTuning.default() if not wavefront else pt.RenderTuning(wavefront_paths=wavefront))
        passes()
        torch.cuda.synchronize()
        for a, b in zip([acc] + imgs, want):
            assert torch.equal(a, b)
    pt.set_tuning(pt.RenderTuning.default())
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        passes()
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            passes()
        for _ in range(3):
            g.replay()
        s.synchronize()
    for a, b in zip([acc] + imgs, want):
        assert torch.equal(a, b)
    ds.close()
