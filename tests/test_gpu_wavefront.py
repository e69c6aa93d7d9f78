"""Wavefronts the library widens to several samples (tuning wavefront_paths =
0): the same images as one sample per wavefront, bit for bit, from one sample
per call to calls that need several widened wavefronts, for single scenes and
batches, and for a pass captured in a CUDA graph (one sample at a time, its
queues untouched by later wide calls)."""
import numpy as np
import pytest
import torch

from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_tuning():
    pt.set_tuning(pt.RenderTuning.default())
    yield
    pt.set_tuning(pt.RenderTuning.default())


def _params(spp):
    return pt.RenderParams(max_depth=4, rr_min_depth=2, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=spp,
                           accumulate=1)


def _render(ds, spp, frame=3):
    n = ds.scene.width * ds.scene.height
    img = torch.zeros(n * 3, device="cuda")
    acc = torch.zeros(n * 3, device="cuda")
    pt.render_pass(ds, _params(spp), frame, img, acc)
    torch.cuda.synchronize()
    return img.cpu().numpy(), acc.cpu().numpy()


# 2^24 paths hold 15 samples of 1100 x 1000 pixels (15.25): 1, 2 and 15 samples
# are one wavefront, 16 are two of 8, 31 three of 11, 11 and 9
@pytest.mark.parametrize("w,h,spp", [(37, 29, 1), (37, 29, 2), (37, 29, 7), (1100, 1000, 15), (1100, 1000, 16),
                                     (1100, 1000, 31)])
def test_widened_wavefronts_render_the_same_image(built, w, h, spp):
    ds = pt.DeviceScene(scenes.tiny_box(w, h, subdiv=2), "cuda")
    got = _render(ds, spp)
    pt.set_tuning(pt.RenderTuning(wavefront_paths=max(1024, w * h)))
    want = _render(ds, spp)
    for g, x in zip(got, want):
        np.testing.assert_array_equal(g, x)
    ds.close()


def test_widened_batch_renders_the_same_images(built):
    dss = [pt.DeviceScene(scenes.tiny_box(w, h, subdiv=2, seed=w), "cuda") for w, h in ((40, 24), (33, 31), (8, 5))]

    def render():
        accs = [torch.zeros(d.scene.width * d.scene.height * 3, device="cuda") for d in dss]
        pt.render_pass_batch(dss, _params(5), 2, None, accs)
        torch.cuda.synchronize()
        return [a.cpu().numpy() for a in accs]

    got = render()
    pt.set_tuning(pt.RenderTuning(wavefront_paths=sum(d.scene.width * d.scene.height for d in dss)))
    for g, x in zip(got, render()):
        np.testing.assert_array_equal(g, x)
    for d in dss:
        d.close()


def test_captured_pass_keeps_its_queues(built):
    ds = pt.DeviceScene(scenes.tiny_box(64, 40, subdiv=2), "cuda")
    n = 64 * 40
    want = _render(ds, 3)
    one = pt.RenderParams(**{**_params(1).__dict__})
    pt.render_pass(ds, one, 0, torch.zeros(n * 3, device="cuda"), torch.zeros(n * 3, device="cuda"))
    torch.cuda.synchronize()
    img, acc = torch.zeros(n * 3, device="cuda"), torch.zeros(n * 3, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        pt.render_pass(ds, _params(3), 3, img, acc)
    _render(ds, 40)          # grows the wide queues after the capture
    acc.zero_()
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(img.cpu().numpy(), want[0])
    np.testing.assert_array_equal(acc.cpu().numpy(), want[1])
    ds.close()
