"""Hash-grid level counts that do not fill a group of gathers (four levels in
training, two in inference): a model's first 2 L features are those of the
16-level model with the same tables, the rest of the hash features is zero;
and table training where most entries are never touched (their moments and
values are not rewritten) in both directions of the sweep."""
import numpy as np
import pytest
import torch

from tests.test_gpu_tuning import _random_queries
from tfg_b200 import nrc

pytestmark = pytest.mark.gpu


def _model(levels, log2=12, seed=3, batch=1024):
    m = nrc.ColorMLP(batch=batch, seed=seed, encoding=nrc.HASHGRID,
                     hashgrid={"n_levels": levels, "log2_hashmap_size": log2})
    m.set_bounds((0, 0, 0), (1, 1, 1))
    return m


@pytest.mark.parametrize("levels", [1, 2, 3, 4, 5, 7, 9, 15])
def test_partial_level_groups(built, levels):
    full, part = _model(16), _model(levels)
    t = (np.random.default_rng(1).random(full.n_table, dtype=np.float32) - 0.5)
    full.set_table(t)
    part.set_table(t[:part.n_table])
    q = _random_queries(500, 4)
    for training in (True, False):
        a = full.encode_features(q, 500, training=training).cpu().numpy()
        b = part.encode_features(q, 500, training=training).cpu().numpy()
        np.testing.assert_array_equal(b[:, :2 * levels], a[:, :2 * levels])
        assert (b[:, 2 * levels:32] == 0).all()
        np.testing.assert_array_equal(b[:, 32:], a[:, 32:])
    full.close()
    part.close()


@pytest.mark.parametrize("log2", [10, 16])
def test_untouched_entries_keep_their_values(built, log2):
    m = _model(16, log2=log2)
    start = m.get_table()
    n = 200
    q = _random_queries(n, 6)
    touched = np.zeros(m.n_table, bool)
    for k in range(3):
        _, g, _ = m.compute_gradient_ex(q, n, seed=k)   # the next step draws with seed k
        touched |= g != 0
        m.train_step(q, n, read_loss=False)
        w, mom, var = (m.get_table(i) for i in (nrc.WEIGHTS, nrc.ADAM_M, nrc.ADAM_V))
        assert (w[~touched] == start[~touched]).all() and (mom[~touched] == 0).all() and (var[~touched] == 0).all()
        assert (w[touched] != start[touched]).mean() > 0.99 and touched.any()
    m.close()
