"""A pass that was run once can be captured: the first call of a process sizes
the queues that the captured call uses, whatever its number of samples, so that
nothing is allocated under capture (which would end it with an error).  Each
case runs in a process of its own, whose queues no other test has sized."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

_FRESH = r"""
import sys
import torch
sys.path.insert(0, sys.argv[1])
from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes
what, w, h, spp = sys.argv[2], int(sys.argv[3]), int(sys.argv[4]), int(sys.argv[5])
sizes = [(w, h)] if what == "pass" else [(w, h), (w // 2, h // 2 + 1)]
dss = [pt.DeviceScene(scenes.tiny_box(x, y, subdiv=2), "cuda") for x, y in sizes]
accs = [torch.zeros(x * y * 3, device="cuda") for x, y in sizes]
imgs = [torch.zeros(x * y * 3, device="cuda") for x, y in sizes]
p = pt.RenderParams(max_depth=4, rr_min_depth=2, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=spp, accumulate=1)

def call():
    if what == "pass":
        pt.render_pass(dss[0], p, 3, imgs[0], accs[0])
    else:
        pt.render_pass_batch(dss, p, 3, imgs, accs)

call()                                    # the only call before the capture is the captured one
torch.cuda.synchronize()
want = [t.clone() for t in accs + imgs]
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    call()
for t in accs:
    t.zero_()
g.replay()
torch.cuda.synchronize()
for a, b in zip(accs + imgs, want):
    assert torch.equal(a, b), "the replayed pass differs"
print("captured")
"""


@pytest.mark.parametrize("what", ["pass", "batch"])
@pytest.mark.parametrize("w,h,spp", [(64, 40, 1), (64, 40, 3), (400, 300, 2)])
def test_first_call_makes_room_for_its_capture(built, what, w, h, spp):
    res = subprocess.run([sys.executable, "-c", _FRESH, str(ROOT), what, str(w), str(h), str(spp)],
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "captured" in res.stdout, res.stdout[-1000:] + res.stderr[-2000:]
