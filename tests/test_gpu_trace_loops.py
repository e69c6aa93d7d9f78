"""Closest-hit loops: small meshes in wavefronts of up to 2^20 paths trace node by
node (step), all others with node and triangle turns.  Work-counting passes
always take turns, so they are the reference on both sides of the rule: images
must be equal bit for bit, also where analytic primitives are not finite."""
import numpy as np
import pytest
import torch

from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes

pytestmark = pytest.mark.gpu


def _both(scene, fmt, depth=5, spp=1):
    ds = pt.DeviceScene(scene, "cuda")
    outs = []
    for profile in (0, pt.PROFILE_COUNTS):
        p = pt.RenderParams(max_depth=depth, rr_min_depth=3, shadow_mesh=1, tri_format=fmt, spp=spp, accumulate=1,
                            profile=profile)
        acc = torch.zeros(scene.width * scene.height * 3, device="cuda")
        pt.render_pass(ds, p, 3, None, acc)
        torch.cuda.synchronize()
        outs.append(acc.cpu().numpy())
    ds.close()
    return outs


# a row more than k_few takes alone, 2^20 paths and one row more; 0, 1, 6,000
# and 6,001 triangles
@pytest.mark.parametrize("w,h", [(256, 257), (1024, 1024), (1024, 1025)])
@pytest.mark.parametrize("ntri", [0, 1, 6000, 6001])
@pytest.mark.parametrize("fmt", [pt.TRIS_REF, pt.TRIS_WATERTIGHT])
def test_step_and_turns_trace_the_same(built, w, h, ntri, fmt):
    base = scenes.box_icosphere(w, h, subdiv=5)
    s = scenes.Scene(base.prims, base.mesh[:ntri], base.lights, base.camera, w, h, bounds=base.bounds)
    got, want = _both(s, fmt)
    assert np.isfinite(want).all() and want.any()
    np.testing.assert_array_equal(got, want)


# k_few alone; beside the long-queue kernels
@pytest.mark.parametrize("w,h", [(40, 33), (300, 256)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_primitives_that_are_not_finite(built, w, h, bad):
    base = scenes.reference_room(w, h, subdiv=2)
    prims = np.concatenate([scenes.sphere_prim((bad, 0.2, -2.0), 0.3, kd=(0.5, 0.4, 0.3)),
                            scenes.sphere_prim((0.1, 0.2, -2.0), bad, kd=(0.5, 0.4, 0.3)),
                            scenes.sphere_prim((0.2, 0.2, -2.0), 0.3, kd=(0.5, 0.4, 0.3)), base.prims])
    s = scenes.Scene(prims, base.mesh, base.lights, base.camera, w, h, bounds=base.bounds)
    got, want = _both(s, pt.TRIS_WATERTIGHT, depth=8)
    assert want.any()
    np.testing.assert_array_equal(got, want)


@pytest.fixture
def default_tuning():
    yield
    pt.set_tuning(pt.RenderTuning.default())


# queues that stay long and queues that become short, on one stream and on two,
# directly and replayed from a graph: the kernels start early either way
@pytest.mark.parametrize("overlap", [0, 1])
@pytest.mark.parametrize("build", [lambda w, h: scenes.box_icosphere(w, h, subdiv=4),
                                   lambda w, h: scenes.spheres_terrain(w, h, subdiv=2, terrain_n=60)])
def test_early_launches_on_one_stream_and_two(built, default_tuning, build, overlap):
    w, h = 400, 301
    s = build(w, h)
    want = _both(s, pt.TRIS_WATERTIGHT, depth=9)[1]
    ds = pt.DeviceScene(s, "cuda")
    p = pt.RenderParams(max_depth=9, rr_min_depth=3, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=1, accumulate=1)
    pt.set_tuning(pt.RenderTuning(overlap_shadow=overlap))
    accs = [torch.zeros(w * h * 3, device="cuda") for _ in range(4)]
    for acc in accs:   # back to back
        pt.render_pass(ds, p, 3, None, acc)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            accs[0].zero_()
            pt.render_pass(ds, p, 3, None, accs[0])
        for _ in range(3):
            graph.replay()
        stream.synchronize()
    for acc in accs:
        np.testing.assert_array_equal(acc.cpu().numpy(), want)
    ds.close()
