"""Device memory that a GPU tree build leaves behind: its result, and at most the
128 MB that the scratch pool keeps -- at once, not after the program has
synchronised another time."""
import ctypes

import numpy as np
import pytest
import torch

from tfg_b200 import _lib, scenes
from tfg_b200.structs import CTinyBVH

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("grid,no_triangles", [(700, False), (700, True)])
def test_build_scratch_goes_back(built, grid, no_triangles):
    mesh = scenes.spheres_terrain(64, 64, subdiv=2, terrain_n=grid).mesh
    n = len(mesh)                                # ~1 M triangles: 0.5 GB of scratch
    if no_triangles:                             # nothing to build: the count's scratch alone, an early exit
        mesh = mesh.copy()
        mesh["tipo"] = 0
    d = torch.from_numpy(mesh.view(np.uint8).copy()).cuda()
    b = CTinyBVH()

    def build(count):
        _lib.call("tfgTinyBVHConstruirGPU", d.data_ptr(), count, ctypes.byref(b), 0)

    build(1000)                                  # what the library loads once
    _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    build(n)
    left = before - torch.cuda.mem_get_info()[0]
    result = 0 if no_triangles else n * (200 + 64 + 48) + (n // 8 + 16) * 80
    assert left <= result + 128 * MB + 32 * MB, (left / MB, result / MB)   # 32 MB: the pool's and cudaMalloc's pages
    _lib.lib.tfgTinyBVHLiberar(ctypes.byref(b))
    assert before - torch.cuda.mem_get_info()[0] <= 160 * MB
