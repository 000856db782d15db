"""Models of different shapes trained from several threads share kernels."""
import threading

import numpy as np
import pytest

from netflix_prize_b200.config import run_lm
from netflix_prize_b200.data import MaskedDataset
from netflix_prize_b200.model import TxModel
from tests.conftest import small_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [((300, 12), (1000, 16)), ((20, 12), (20, 64)), ((200, 12), (200, 64))])
def test_two_threads_train_models_of_two_shapes(shapes):
    """Each shape's kernels need another amount of shared memory; each thread's model
    is, bit for bit, the one trained alone."""
    tr, pr = small_sets(n_users=200, n_items=120, n_train=4000, seed=5)
    cfgs = [run_lm(f, 2, n_time_bins=30).replace(n_freq_bins=bins) for f, bins in shapes]
    alone, models, errors = [], [], []
    for c in cfgs:
        a = TxModel(tr, MaskedDataset(pr), c)
        for e in range(1, 401):
            a.fit_epoch(tr, pr, e)
        alone.append(np.asarray(a.get_param("ifeat"), np.float32))
        models.append(TxModel(tr, MaskedDataset(pr), c))

    def train(m):
        try:
            for e in range(1, 401):
                m.fit_epoch(tr, pr, e)
        except Exception as x:  # noqa: BLE001
            errors.append(x)

    threads = [threading.Thread(target=train, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for m, a in zip(models, alone):
        b = np.asarray(m.get_param("ifeat"), np.float32)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
