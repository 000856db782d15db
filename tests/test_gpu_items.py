"""Rules of the item stratum that its parity on ordinary data does not show."""
import numpy as np
import pytest
import torch

from netflix_prize_b200.abi import PREC_BF16_READ_ALL
from netflix_prize_b200.config import OrdinalHeadConfig, run_lm
from netflix_prize_b200.data import Dataset, MaskedDataset
from netflix_prize_b200.model import TxModel
from oracle import pyoracle as po
from tests.test_gpu_chains import ITEM_COUNTS, counted_items

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


def long_items(counts):
    """Item k is rated by the first counts[k] users, each rating on a day of its own
    (one frequency bin); a query pair a user."""
    n = max(counts)
    u = np.concatenate([np.arange(c) for c in counts])
    i = np.repeat(np.arange(len(counts)), counts)
    o = np.lexsort((i, u))
    u, i = u[o], i[o]
    tr = Dataset.from_ratings(u, i, 1 + (u * 7 + i * 3) % 5, 100 * (i + 1) + u % 50, n, len(counts) + 1, "long")
    pr = Dataset.from_ratings(np.arange(n), np.full(n, len(counts)), np.full(n, 3), np.full(n, 900), n, len(counts) + 1,
                              "long_pr")
    return tr, pr


@pytest.mark.parametrize("f", [32])
def test_decay_does_not_depend_on_the_block_threshold(f):
    """Items of 32,768 ratings and more decay by factors rounded to FP32 (5.96e-8 here),
    shorter ones by the exact ones (3.5e-8), whichever of the two paths takes them.

    Tolerance: an item's row is rounded at most once a rating, half an ulp each way:
    sqrt(40000) 2^-25 = 6e-6 of the row, four times that for the largest of 32 columns.
    The other factor would be 5000 x 2.4e-8 = 1.2e-4 off in the shortest item."""
    counts = [40000, 32767, 5000]
    tr, pr = long_items(counts)
    zero = {k: 0.0 for k in ("lr_u", "lr_u2", "lr_ub", "lr_ubd", "lr_y", "lr_yb", "lr_ta", "lr_tu", "lr_cu", "lr_ib",
                             "lr_ti", "lr_ibf")}
    cfg = run_lm(f, 1, n_time_bins=30).replace(lr_i=5e-6, reg_i=0.007, lr_iqf=5e-6, reg_iqf=0.007, **zero)
    rng = np.random.default_rng(4)
    init = {"ufeat": rng.normal(0, 1 / np.sqrt(f), (max(counts), f)).astype(np.float32),
            "ifeat": rng.normal(0, 0.3, (4, f)).astype(np.float32),
            "ifeat_freq": rng.normal(0, 0.3, (4 * cfg.n_freq_bins, f)).astype(np.float32),
            "yfeat": np.zeros((4, f), np.float32)}
    lr, reg = float(np.float32(5e-6)), float(np.float32(0.007))
    rounded = float(np.float32(1.0 - lr * reg))
    assert abs(rounded - (1.0 - 2.0 ** -24)) < 1e-12
    want = []
    for heavy in (0, 1, 4096, 100000):
        m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=heavy)
        for n, v in init.items():
            m.set_param(n, v)
        m.fit_epoch(tr, pr, 1)
        if not want:
            p, g = init["ufeat"].astype(np.float64), float(np.asarray(m.get_param("gbias")).ravel()[0])
            for k, c in enumerate(counts):
                a = rounded if c >= 32768 else 1.0 - lr * reg
                q, h = init["ifeat"][k].astype(np.float64), init["ifeat_freq"][k * cfg.n_freq_bins].astype(np.float64)
                for x, y in zip(p[:c], 1 + (np.arange(c) * 7 + k * 3) % 5):
                    d = lr * (g + x @ (q + h) - y) * x
                    q, h = a * q - d, a * h - d
                want.append((q, h))
        q, h = m.get_param("ifeat"), m.get_param("ifeat_freq").reshape(4, cfg.n_freq_bins, f)[:, 0]
        for k in range(3):
            for got, w in ((q[k], want[k][0]), (h[k], want[k][1])):
                assert np.max(np.abs(got - w)) < 2.4e-5 * np.max(np.abs(w)), (heavy, k)


@pytest.mark.parametrize("f", [32, 160])
def test_thresholds_that_take_the_same_items_give_the_same_bits(f):
    """Every item here has more than 4,096 ratings. Above 128 columns items of 32,768
    ratings take a block at any threshold."""
    tr, pr = long_items([40000, 32767, 5000])
    cfg = run_lm(f, 1, n_time_bins=30)
    for same in ((0, 1, 4096), (32768, 40000, 100000) if f > 128 else (32768, 40000)):
        got = []
        for heavy in same:
            m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=heavy)
            m.fit_epoch(tr, pr, 1)
            got.append({n: np.asarray(m.get_param(n), np.float32).view(np.uint32) for n in ITEM_PARAMS})
        for g in got[1:]:
            for n in ITEM_PARAMS:
                assert np.array_equal(g[n], got[0][n]), (same, n)


FROZEN = {n: 0.0 for n in ("lr_u", "lr_u2", "lr_ub", "lr_ubd", "lr_y", "lr_yb", "lr_ta", "lr_tu", "lr_cu")}
ROUND_COUNTS = [64, 32, 20, 2]


def one_bin_rounds():
    """Item k is rated by the first ROUND_COUNTS[k] of 64 users, each rating in a time
    bin of its own (of 64) and in frequency bin 0."""
    u = np.concatenate([np.arange(c) for c in ROUND_COUNTS])
    i = np.repeat(np.arange(len(ROUND_COUNTS)), ROUND_COUNTS)
    o = np.lexsort((i, u))
    u, i = u[o], i[o]
    n = len(ROUND_COUNTS) + 1
    tr = Dataset.from_ratings(u, i, 1 + (u * 7 + i * 3) % 5, 20 * u + i, 64, n, "rounds")
    pr = Dataset.from_ratings(np.arange(64), np.full(64, n - 1), np.full(64, 3), 20 * np.arange(64) + 19, 64, n, "rounds_pr")
    return tr, pr


def chain_errors(p, q, h, y, lr, g, th):
    """The errors of an item's ratings, one after another in 64 bits."""
    out = []
    for x, t in zip(p, y):
        e = g + x @ (q + h) - t
        if th is not None:
            c = np.concatenate([[0.0], 1 / (1 + np.exp(-(th - (e + t)))), [1.0]])
            e = 1.0 - c[t] - c[t - 1]
        q, h = q - lr * e * x, h - lr * e * x
        out.append(e)
    return np.array(out)


@pytest.mark.parametrize("f,low_memory,ordinal", [(32, True, False), (64, True, False), (96, True, False), (128, True, False),
                                                  (160, True, False), (224, True, False), (256, True, False),
                                                  (20, False, False), (160, False, False), (256, False, False),
                                                  (20, True, True), (128, True, True), (200, True, True)])
def test_a_round_keeps_the_digits_of_its_rows(f, low_memory, ordinal):
    """Rows of equal values and steps of the size of 1 / |row|^2, where what a product of
    two rows loses is lost in every column alike and moves the next rating's error by
    as much. The errors are read from the time-bin biases, one a rating (lr_ti = 1).

    Tolerance: a score of up to 4 comes from some 20 roundings (a lane's share of the
    columns, five or six levels of sums, the biases, the system's row), half an ulp,
    2.4e-7, each: 4.8e-6. The head's gradient has half that slope at most, but is a
    quotient by a probability above 0.05 of three roundings of 6e-8: 2.4e-6 + 3.6e-6.
    Products of two 8-bit parts of each value are 1.8e-5 (with the head) and 7e-5 off."""
    tr, pr = one_bin_rounds()
    names = ("lr_u", "lr_u2", "lr_ud", "lr_ub", "lr_ubd", "lr_y", "lr_yb", "lr_yd", "lr_ta", "lr_tu", "lr_cu", "lr_ib", "lr_ibf",
             "reg_i", "reg_iqf")
    value = np.float32(1.003898)  # 2^-8 and 2^-17 past a number of 8 bits
    lr = float(np.float32((1.2 if ordinal else 0.45) / (f * float(value) ** 2)))
    th = (0.5, 1.25, 3.75, 5.5)
    cfg = run_lm(f, 1, n_time_bins=64, low_memory=low_memory).replace(
        lr_i=lr, lr_iqf=lr, lr_ti=1.0, ordinal_head=OrdinalHeadConfig(th, 0.001, 0.0, 0.0) if ordinal else None,
        **{n: 0.0 for n in names})
    n, nf = tr.n_items, cfg.n_freq_bins
    rng = np.random.default_rng(6)
    init = {"ufeat": np.full((64, f), value, np.float32), "ufeat2": np.zeros((64, f), np.float32),
            "ifeat": rng.normal(0, 0.01, (n, f)).astype(np.float32), "yfeat": np.zeros((n, f), np.float32),
            "ifeat_freq": rng.normal(0, 0.01, (n * nf, f)).astype(np.float32)}
    if not low_memory:
        init["yfeat_day"] = np.zeros((n, f), np.float32)
    for heavy in (1, 100000):
        m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=heavy)
        for k, v in init.items():
            m.set_param(k, v)
        m.fit_epoch(tr, pr, 1)
        assert np.array_equal(m.get_param("ufeat"), init["ufeat"])
        g = float(np.asarray(m.get_param("gbias")).ravel()[0])
        got = -np.asarray(m.get_param("bit_bin"), np.float64).reshape(n, 64)
        for k, c in enumerate(ROUND_COUNTS):
            y = 1 + (np.arange(c) * 7 + k * 3) % 5
            want = chain_errors(init["ufeat"][:c].astype(np.float64), init["ifeat"][k].astype(np.float64),
                                init["ifeat_freq"][k * nf].astype(np.float64), y, lr, g, np.array(th) if ordinal else None)
            assert np.max(np.abs(got[k, :c] - want)) < (6e-6 if ordinal else 4.8e-6), (heavy, c)


@pytest.mark.parametrize("f,low_memory", [(20, True), (64, True), (128, True), (160, True), (256, True), (60, False),
                                          (200, False)])
def test_rows_far_beyond_the_learning_rate(f, low_memory):
    """Values of 100 sqrt(2 / lr), far past what FP16 holds without a scale: the second
    rating's error is that of the 64-bit chain.

    Tolerance: relative, all terms of a score and of a dot have one sign; 20 roundings of
    2^-24 a score, as many for the first error's way into the second, 64 + 8 for the dot
    of the rows: 112 x 2^-24 = 7e-6."""
    u, i = np.array([0, 0, 1, 1, 63]), np.array([0, 1, 0, 1, 2])
    tr = Dataset.from_ratings(u, i, 1 + (u + i) % 5, 20 * u + i, 64, 4, "large")
    pr = Dataset.from_ratings(np.arange(64), np.full(64, 3), np.full(64, 3), 20 * np.arange(64) + 9, 64, 4, "large_pr")
    lr = float(np.float32(0.005))
    cfg = run_lm(f, 1, n_time_bins=64, low_memory=low_memory).replace(
        lr_i=lr, lr_iqf=lr, lr_ti=1.0, lr_ib=0.0, lr_ibf=0.0, lr_ud=0.0, lr_yd=0.0, reg_i=0.0, reg_iqf=0.0, **FROZEN)
    rng = np.random.default_rng(7)
    nf = cfg.n_freq_bins
    init = {"ufeat": np.full((64, f), 2000.0, np.float32), "ufeat2": np.zeros((64, f), np.float32),
            "ifeat": rng.uniform(0.01, 0.02, (4, f)).astype(np.float32), "yfeat": np.zeros((4, f), np.float32),
            "ifeat_freq": rng.uniform(0.01, 0.02, (4 * nf, f)).astype(np.float32)}
    if not low_memory:
        init["yfeat_day"] = np.zeros((4, f), np.float32)
    for heavy in (1, 100000):
        m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=heavy)
        for k, v in init.items():
            m.set_param(k, v)
        m.fit_epoch(tr, pr, 1)
        g = float(np.asarray(m.get_param("gbias")).ravel()[0])
        got = -np.asarray(m.get_param("bit_bin"), np.float64).reshape(4, 64)
        for k in range(2):
            y = 1 + (np.arange(2) + k) % 5
            want = chain_errors(init["ufeat"][:2].astype(np.float64), init["ifeat"][k].astype(np.float64),
                                init["ifeat_freq"][k * nf].astype(np.float64), y, lr, g, None)
            assert np.max(np.abs(got[k, :2] / want - 1)) < 7e-6, (heavy, k)


# strong updates and decays of rows and bins, as in the tests of the item stratum without the head
STRONG = dict(lr_ti=0.002, lr_ibf=0.003, lr_iqf=0.004, reg_iqf=0.05, reg_i=0.05, sigma_u=0.1, sigma_i=0.1, sigma_iqf=0.1)


@pytest.mark.parametrize("heavy", [1, 40, 100000])
@pytest.mark.parametrize("f", [20, 64, 96, 160, 256])
def test_item_stratum_with_the_ordinal_head(f, heavy):
    """Items in rounds and by pairs against their chains in 64 bits (src/tsvdx4p.rs:644-762
    with the head's gradient, src/lib.rs:562-598), users frozen; the bound of one epoch's
    parity, 2e-5."""
    tr, pr = counted_items(ITEM_COUNTS, 200, 5)
    th = np.array([0.5, 1.25, 3.75, 5.5])
    cfg = run_lm(f, 1, n_time_bins=48).replace(ordinal_head=OrdinalHeadConfig(tuple(th), 0.001, 0.0, 0.0), **STRONG, **FROZEN)
    m = TxModel(tr, MaskedDataset(pr), cfg, heavy_item_ratings=heavy)
    rng = np.random.default_rng(8)
    m.set_param("ufeat2", rng.normal(0, 0.05, (200, f)).astype(np.float32))
    names = ["ufeat", "ufeat2", "tu_mean"] + ITEM_PARAMS
    P = {n: np.asarray(m.get_param(n), np.float64) for n in names}
    m.fit_epoch(tr, pr, 1)
    yc, ycb = np.asarray(m.get_param("ycache"), np.float64), np.asarray(m.get_param("ycache_bias"), np.float64)
    g = float(np.asarray(m.get_param("gbias")).ravel()[0])
    n, nf, T = tr.n_items, cfg.n_freq_bins, cfg.n_time_bins
    qf, bt, bf = P["ifeat_freq"].reshape(n, nf, f), P["bit_bin"].reshape(n, T), P["ibias_freq"].reshape(n, nf)
    q, ib = P["ifeat"].reshape(n, f), P["ibias"].ravel()
    _, at, day_cnt = np.unique(np.concatenate([tr.user_idxs, pr.user_idxs]) * 10000
                               + np.concatenate([tr.dates, pr.dates]).astype(np.int64), return_inverse=True, return_counts=True)
    fbin = np.minimum(np.log2(day_cnt[at[:len(tr.user_idxs)]]).astype(int), nf - 1)
    assert len(np.unique(fbin)) > 2
    day_range = int(max(tr.dates.max(), pr.dates.max())) + 1
    for i in range(n):
        rows = np.nonzero(tr.item_idxs == i)[0]
        for t in rows[np.argsort(tr.user_idxs[rows], kind="stable")]:
            u, day, b = tr.user_idxs[t], int(tr.dates[t]), fbin[t]
            tb = min(day * T // day_range, T - 1)
            dt = day - P["tu_mean"][u]
            dv = np.sign(dt) * abs(dt) ** np.float64(np.float32(cfg.beta))
            pe = P["ufeat"][u] + yc[u] + dv * P["ufeat2"][u]
            x = g + ycb[u] + ib[i] + bt[i, tb] + bf[i, b] + pe @ (q[i] + qf[i, b])
            c = np.concatenate([[0.0], 1 / (1 + np.exp(-(th - x))), [1.0]])
            y = int(tr.raw_ratings[t])
            e = (c[y] * (1 - c[y]) - c[y - 1] * (1 - c[y - 1])) / max(c[y] - c[y - 1], 1e-6)
            ib[i] -= cfg.lr_ib * e
            bt[i, tb] -= cfg.lr_ti * e
            bf[i, b] -= cfg.lr_ibf * e
            q[i], qf[i, b] = (q[i] - cfg.lr_i * (e * pe + cfg.reg_i * q[i]),
                              qf[i, b] - cfg.lr_iqf * (e * pe + cfg.reg_iqf * qf[i, b]))
    for name, want in (("ifeat", q), ("ifeat_freq", qf), ("ibias", ib), ("bit_bin", bt), ("ibias_freq", bf)):
        assert np.max(np.abs(np.asarray(m.get_param(name), np.float64).ravel() - want.ravel())) < 2e-5, name


@pytest.mark.parametrize("heavy", [1, 40, 100000])
@pytest.mark.parametrize("f", [20, 64, 128, 160, 256])
def test_item_stratum_with_rounded_user_rows(f, heavy):
    """User rows that are BF16 numbers already: the precision form that reads them as
    such is, users frozen, within the bound of FP32 parity of the oracle's epoch."""
    tr, pr = counted_items(ITEM_COUNTS, 200, 5)
    cfg = run_lm(f, 1, n_time_bins=48).replace(**STRONG, **FROZEN)
    rng = np.random.default_rng(9)
    init = {n: torch.as_tensor(rng.normal(0, sd, (200, f)), dtype=torch.bfloat16).float().numpy()
            for n, sd in (("ufeat", 0.1), ("ufeat2", 0.05))}
    init["yfeat"] = np.zeros((tr.n_items, f), np.float32)
    o = po.OracleModel(tr, MaskedDataset(pr), cfg)
    m = TxModel(tr, MaskedDataset(pr), cfg, precision=PREC_BF16_READ_ALL, heavy_item_ratings=heavy)
    for n, v in init.items():
        o.set_param(n, v)
        m.set_param(n, v)
    o.fit_epoch(1, po.SCHED_P, nsvd_norm_exp=1.0, n_threads=1)
    m.fit_epoch(tr, pr, 1)
    assert np.array_equal(m.get_param("ufeat"), init["ufeat"])
    for n in ITEM_PARAMS:
        a, b = np.asarray(m.get_param(n), np.float64).ravel(), np.asarray(o.get_param(n), np.float64).ravel()
        assert np.max(np.abs(a - b) - 1e-5 * np.abs(b)) < 2e-5, n
