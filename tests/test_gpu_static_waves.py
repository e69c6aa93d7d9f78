"""The allocation-free entry point where its 16,384 paths of scratch are not a
whole number of samples: images equal to the allocating entry point's, bit for
bit."""
import numpy as np
import pytest
import torch

from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(128, 100, 3), (127, 129, 2), (33, 31, 17), (128, 128, 2), (1, 1, 5)])
def test_wavefronts_that_split_samples(built, w, h, spp):
    ds = pt.DeviceScene(scenes.box_icosphere(w, h, subdiv=3), "cuda")
    p = pt.RenderParams(max_depth=6, rr_min_depth=3, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=spp, accumulate=1)
    outs = []
    for render in (pt.render_pass_static, pt.render_pass):
        img = torch.zeros(w * h * 3, device="cuda")
        acc = torch.zeros(w * h * 3, device="cuda")
        render(ds, p, 4, img, acc)
        torch.cuda.synchronize()
        outs.append((img.cpu().numpy(), acc.cpu().numpy()))
    assert np.isfinite(outs[1][1]).all()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    ds.close()
