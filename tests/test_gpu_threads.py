"""Host threads that render on one stream with different numbers of samples: the
calls need queues of different sizes, and a call that grows them must not free
those of a call on another thread that has still to enqueue its launches.  In a
process of its own, whose queues start empty, so that most calls grow them."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

_FRESH = r"""
import sys
import threading
import torch
sys.path.insert(0, sys.argv[1])
from tfg_b200 import pathtracer as pt
from tfg_b200 import scenes
W, H = 120, 90
ds = pt.DeviceScene(scenes.tiny_box(W, H, subdiv=2), "cuda")

def render(spp, frame, acc):
    p = pt.RenderParams(max_depth=4, rr_min_depth=2, shadow_mesh=1, tri_format=pt.TRIS_WATERTIGHT, spp=spp, accumulate=1)
    pt.render_pass(ds, p, frame, None, acc)

jobs = [[(spp, 100 * t + spp) for spp in range(1 + t, 25, 2)] for t in range(3)]
out = [[torch.zeros(W * H * 3, device="cuda") for _ in j] for j in jobs]
torch.cuda.synchronize()
start, errors = threading.Barrier(3), []

def work(t):
    try:
        start.wait()
        for (spp, frame), acc in zip(jobs[t], out[t]):
            render(spp, frame, acc)
    except Exception as e:
        errors.append(e)

threads = [threading.Thread(target=work, args=(t,)) for t in range(3)]
for t in threads: t.start()
for t in threads: t.join()
torch.cuda.synchronize()
assert not errors, errors
for j, o in zip(jobs, out):
    for (spp, frame), acc in zip(j, o):
        want = torch.zeros_like(acc)
        render(spp, frame, want)
        torch.cuda.synchronize()
        assert torch.equal(acc, want), (spp, frame)
print("equal")
"""


def test_threads_with_different_sample_counts(built):
    res = subprocess.run([sys.executable, "-c", _FRESH, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "equal" in res.stdout, res.stdout[-1000:] + res.stderr[-2000:]
