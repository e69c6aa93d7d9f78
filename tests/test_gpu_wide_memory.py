"""Device memory of widened wavefronts: at most an eighth of what is free, asked
for once, and given back when a tuning names a wavefront size.  Run in processes of their own, whose queues start empty."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

_COMMON = r"""
import sys
import torch
sys.path.insert(0, sys.argv[1])
from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes
W, H = 600, 500
PATH = 224                                     # bytes of queues and state per path
ds = pt.DeviceScene(scenes.tiny_box(W, H, subdiv=2), "cuda")
accs = [torch.zeros(W * H * 3, device="cuda") for _ in range(6)]
p = pt.RenderParams(max_depth=4, rr_min_depth=2, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=8, accumulate=1)

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

def taken(k):
    before = free()
    pt.render_pass(ds, p, 5, None, accs[k])
    return before - free()

MB = 1 << 20
wide = W * H * 8 * PATH                        # all eight samples in one wavefront
one = pt.RenderParams(**{**p.__dict__, "spp": 1})
pt.render_pass(ds, one, 5, None, accs[5])      # the ordinary queues, and whatever the library loads once
"""

# 2 GB left: an eighth of them holds three samples; 2 GB more change nothing
# until the tuning is set again
_BOUNDED = _COMMON + r"""
extra = torch.empty(2048 * MB, dtype=torch.uint8, device="cuda")
filler = torch.empty(free() - 2048 * MB, dtype=torch.uint8, device="cuda")
first = taken(0)
assert 0 < first <= 2048 * MB // 8 + 16 * MB, first
del extra
torch.cuda.empty_cache()
assert abs(taken(1)) <= 16 * MB
pt.set_tuning(pt.RenderTuning.default())
again = taken(2)
assert again > 16 * MB, again
del filler
torch.cuda.empty_cache()
pt.set_tuning(pt.RenderTuning.default())
taken(3)
for k in (1, 2, 3):
    assert torch.equal(accs[0], accs[k])
print("fine")
"""


_GIVEN_BACK = _COMMON + r"""
before = free()
assert taken(0) >= wide
pt.set_tuning(pt.RenderTuning.default())
assert before - free() >= wide                 # still the library's choice of size
pt.set_tuning(pt.RenderTuning(wavefront_paths=W * H))
assert before - free() <= 16 * MB, before - free()
taken(1)
pt.set_tuning(pt.RenderTuning.default())
assert taken(2) >= wide
for k in (1, 2):
    assert torch.equal(accs[0], accs[k])
print("fine")
"""


def _run(code):
    res = subprocess.run([sys.executable, "-c", code, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "fine" in res.stdout, res.stdout[-1000:] + res.stderr[-2000:]


def test_bounded_by_free_memory_and_asked_once(built):
    _run(_BOUNDED)


def test_given_back_with_a_named_size(built):
    _run(_GIVEN_BACK)
