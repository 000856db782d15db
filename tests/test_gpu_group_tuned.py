"""The autotuned thresholds of a stratified group's item strata."""
import numpy as np
import pytest

from netflix_prize_b200.config import run_lm
from netflix_prize_b200.data import Dataset, MaskedDataset
from netflix_prize_b200.model import TxGroup, TxModel
from tests.test_gpu_parity import PARAMS

pytestmark = pytest.mark.gpu


def even_items(n_users, n_items, per_user):
    """Every item has about n_users per_user / n_items ratings; a query pair a user."""
    rng = np.random.default_rng(2)
    pick = np.argsort(rng.random((n_users, n_items)), axis=1)[:, :per_user + 1]
    u, i = np.repeat(np.arange(n_users), per_user), np.sort(pick[:, :per_user], axis=1).ravel()
    tr = Dataset.from_ratings(u, i, rng.integers(1, 6, len(u)), rng.integers(0, 900, len(u)), n_users, n_items, "even")
    o = np.argsort(pick[:, -1], kind="stable")
    pr = Dataset.from_ratings(o, pick[o, -1], rng.integers(1, 6, n_users), rng.integers(0, 900, n_users), n_users, n_items,
                              "even_pr")
    return tr, pr


@pytest.mark.parametrize("n_users,n_items,per_user", [(3500, 60, 50), (7500, 40, 30), (12000, 30, 25)])
def test_tuned_variants_equal_single_models_and_do_not_fall_behind(n_users, n_items, per_user):
    """Items of 2,900, 5,600 and 10,000 ratings on sets whose own threshold is a few
    hundred: the smallest are below every constant that is tried, and rounds take a
    fraction of a one-warp chain's time for all of them (nowhere near the 1.5 that is
    allowed for here). The group and single models of its thresholds share all bits."""
    tr, pr = even_items(n_users, n_items, per_user)
    cfgs = [run_lm(f, 3, n_time_bins=30, seed=f) for f in (20, 60, 200)]

    def epoch_ms(g):
        g.fit_epoch(1)
        best = 1e9
        for e in (2, 3, 4):
            g.fit_epoch(e)
            best = min(best, g.last_epoch_ms())
        return best

    plain, tuned = TxGroup(tr, MaskedDataset(pr), cfgs), TxGroup(tr, MaskedDataset(pr), cfgs)
    thr = [int(t) for t in tuned.autotune()]
    t_plain, t_tuned = epoch_ms(plain), epoch_ms(tuned)
    assert t_tuned < 1.5 * t_plain, (thr, t_plain, t_tuned)
    for c, t, gm in zip(cfgs, thr, tuned.models):
        m = TxModel(tr, MaskedDataset(pr), c, heavy_item_ratings=t)
        for e in (1, 2, 3, 4):
            m.fit_epoch(tr, pr, e)
        for n in PARAMS:
            a, b = np.asarray(gm.get_param(n), np.float32), np.asarray(m.get_param(n), np.float32)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (t, n)
