"""Training steps queued one behind the other give what the same steps give one
at a time, bit for bit: the kernels of a step start before their predecessors
have ended, and every one of them must still see all that was written before
it (gradients, moments, masters, the step's time).

Table gradients are float atomics, whose order is not fixed.  The tables here
are fine enough (64 cells per axis and more) and the batch small enough (128
samples) that hardly an entry gets three contributions of one step -- the
expected number is below 0.02 over all levels and steps -- and a sum of two
does not depend on their order."""
import numpy as np
import pytest
import torch

from tests.test_gpu_tuning import _random_queries
from tfg_b200 import nrc

pytestmark = pytest.mark.gpu
STEPS = 4
FINE = {"n_levels": 5, "log2_hashmap_size": 19, "base_resolution": 64.0, "per_level_scale": 1.5}


def _train(encoding, width, layers, batch, rows, n, wait):
    m = nrc.ColorMLP(batch=batch, seed=7, hidden_layers=layers, width=width, encoding=encoding,
                     hashgrid=FINE if encoding == nrc.HASHGRID else None)
    m.set_bounds((0, 0, 0), (1, 1, 1))
    if encoding == nrc.HASHGRID:
        m.set_table(np.random.default_rng(2).random(m.n_table, dtype=np.float32) - np.float32(0.5))
    for _ in range(STEPS):
        m.train_step(rows, n, read_loss=False)
        if wait:
            torch.cuda.synchronize()
    assert m.state()["adam_t"] == STEPS
    out = [m.get_params(k) for k in range(4)]
    if encoding == nrc.HASHGRID:
        out += [m.get_table(k) for k in range(4)]
    m.close()
    return out


@pytest.mark.parametrize("encoding,width,layers,batch", [
    (nrc.FREQUENCY, 64, 5, 128), (nrc.FREQUENCY, 64, 3, 16384), (nrc.FREQUENCY, 128, 7, 128 * 160),
    (nrc.HASHGRID, 64, 5, 128), (nrc.HASHGRID, 128, 3, 128)])
def test_queued_steps_equal_single_steps(built, encoding, width, layers, batch):
    n = 50000
    rows = _random_queries(n, 11)
    want = _train(encoding, width, layers, batch, rows, n, wait=True)
    for _ in range(2):
        for a, b in zip(_train(encoding, width, layers, batch, rows, n, wait=False), want):
            np.testing.assert_array_equal(a, b)
