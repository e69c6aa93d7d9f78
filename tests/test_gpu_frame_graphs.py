"""Frames of several renderers in turn, each captured behind another's graph: the
executable graph is updated where the shape is the same (other buffers, sizes and
scenes) and built anew where it is not (another depth, other steps).  Images are
those of frames without graphs, bit for bit."""
import numpy as np
import pytest
import torch

from tfg_b200 import nrc
from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes

pytestmark = pytest.mark.gpu


def _frames(use_graph, order):
    dss, rends = [], []
    st = torch.cuda.Stream()
    # short wavefronts alone on their kernel, long ones of two sizes, another depth
    for w, h, depth, build in ((64, 48, 5, scenes.tiny_box), (320, 240, 5, scenes.box_icosphere),
                               (400, 240, 5, scenes.box_icosphere), (320, 240, 8, scenes.box_icosphere)):
        s = build(w, h, subdiv=3)
        ds = pt.DeviceScene(s, "cuda")
        mlp = nrc.ColorMLP(seed=7)
        mlp.set_bounds(*s.bounds)
        p = pt.RenderParams(max_depth=depth, rr_min_depth=3, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT)
        rends.append(nrc.NrcRenderer(ds, mlp, p, train_steps=0, use_graph=use_graph, stream=st))
        dss.append(ds)
    got = []
    for k, i in enumerate(order):
        with torch.cuda.stream(st):
            rends[i].frame(k)
        st.synchronize()
        got.append(rends[i].img.cpu().numpy().copy())
    for ds in dss:
        ds.close()
    return got


@pytest.mark.parametrize("order", [(0, 1, 2, 1, 2, 2, 3, 1, 0, 3), (3, 3, 0, 0, 2, 1, 1, 2)])
def test_renderers_in_turn(built, order):
    want, got = _frames(False, order), _frames(True, order)
    for g, w in zip(got, want):
        assert w.any()
        np.testing.assert_array_equal(g, w)
