"""Rules of the item stratum that its parity on ordinary data does not show."""
import numpy as np
import pytest
import torch

from netflix_prize_b200.config import OrdinalHeadConfig, run_lm
from netflix_prize_b200.data import Dataset, MaskedDataset
from netflix_prize_b200.model import TxModel

pytestmark = pytest.mark.gpu

ITEM_PARAMS = ["ifeat", "ifeat_freq", "ibias", "bit_bin", "ibias_freq"]


def two_groups(n_a, n_b, seed):
    """n_a items of 40 ratings each and n_b of 33, rated by two groups of 60 users
    with no item in common; a query pair a user on an unrated item of its group."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([(60 if k >= n_a else 0) + rng.choice(60, size=33 if k >= n_a else 40, replace=False)
                        for k in range(n_a + n_b)])
    i = np.repeat(np.arange(n_a + n_b), [40] * n_a + [33] * n_b)
    o = np.lexsort((i, u))
    u, i = u[o], i[o]
    tr = Dataset.from_ratings(u, i, rng.integers(1, 6, len(u)), rng.integers(0, 900, len(u)), 120, n_a + n_b + 2, "groups")
    pu = np.arange(120)
    pr = Dataset.from_ratings(pu, n_a + n_b + (pu >= 60), rng.integers(1, 6, 120), rng.integers(0, 900, 120), 120,
                              n_a + n_b + 2, "groups_pr")
    return tr, pr


@pytest.mark.parametrize("f,low_memory,ordinal", [(33, True, False), (96, True, False), (70, False, False),
                                                  (130, False, False), (160, True, True), (200, True, True),
                                                  (256, True, False)])
def test_a_row_that_is_not_finite_stays_with_its_item(f, low_memory, ordinal):
    """Every block's first item has a row that is not finite, its later ones share no
    rater with those: they are, bit for bit, what they are beside finite rows."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tr, pr = two_groups(sms, 2 * sms, 3)
    cfg = run_lm(f, 1, n_time_bins=30, low_memory=low_memory).replace(
        ordinal_head=OrdinalHeadConfig((0.5, 1.25, 3.75, 5.5), 0.001, 0.0, 0.0) if ordinal else None)
    got = []
    for bad in (False, True):
        m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=1)
        if bad:
            q = m.get_param("ifeat").copy()
            q[np.arange(sms), np.arange(sms) % f] = np.resize([np.nan, np.inf, -np.inf], sms)
            m.set_param("ifeat", q)
        m.fit_epoch(tr, pr, 1)
        got.append({n: np.asarray(m.get_param(n), np.float32).reshape(sms * 3 + 2, -1) for n in ITEM_PARAMS})
    assert not np.isfinite(got[1]["ifeat"][:sms]).all(1).any()
    for n in ITEM_PARAMS:
        assert np.isfinite(got[0][n]).all(), n
        assert np.array_equal(got[1][n][sms:], got[0][n][sms:]), n
