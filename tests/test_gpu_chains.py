"""The strata's blocked chains at the sizes where they can go wrong, against the
oracle's tsvdx4p epoch (the reference's src/tsvdx4p.rs:390-762).

Tolerance: a parameter is a sum of at most a few hundred updates of at most
|lr x| ~ 1e-2 each, in FP32 in both, in another order; 2e-5 absolute is the
bound every other parity test of one epoch holds.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from netflix_prize_b200.abi import PREC_FP32
from netflix_prize_b200.config import OrdinalHeadConfig, run_lm
from netflix_prize_b200.data import Dataset, MaskedDataset
from netflix_prize_b200.encoder import foldin
from netflix_prize_b200.model import TxModel
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

PARAMS = ["ubias", "ibias", "ufeat", "ufeat2", "ifeat", "yfeat", "alpha_u", "but_bin", "bit_bin", "ybias",
          "ubias_day", "ibias_freq", "ifeat_freq", "cu", "cut"]


def counted_sets(counts, n_items, seed):
    """Users with exactly these numbers of training ratings, several on a day,
    and two query pairs each."""
    rng = np.random.default_rng(seed)
    u, i, d, pu, pi, pd = [], [], [], [], [], []
    for k, n in enumerate(counts):
        items = np.sort(rng.choice(n_items, size=n + 2, replace=False))
        days = rng.integers(0, 1500, size=max(1, n // 3))
        q = rng.permutation(n + 2)
        u += [k] * n
        i += list(items[np.sort(q[:n])])
        d += list(rng.choice(days, size=n))
        pu += [k] * 2
        pi += list(items[q[n:]])
        pd += list(rng.choice(days, size=2))
    tr = Dataset.from_ratings(u, i, rng.integers(1, 6, len(u)), d, len(counts), n_items, "counted_tr")
    o = np.lexsort((np.array(pu), np.array(pi)))
    pr = Dataset.from_ratings(np.array(pu)[o], np.array(pi)[o], rng.integers(1, 6, len(pu)), np.array(pd)[o],
                              len(counts), n_items, "counted_pr")
    return tr, pr


def check_epochs(tr, pr, cfg, epochs=2, **kw):
    o = po.OracleModel(tr, MaskedDataset(pr), cfg)
    g = TxModel(tr, MaskedDataset(pr), cfg, precision=PREC_FP32, **kw)
    for e in range(1, epochs + 1):
        o.fit_epoch(e, po.SCHED_P, nsvd_norm_exp=1.0, n_threads=1)
        g.fit_epoch(tr, pr, e)
    names = PARAMS if cfg.low_memory else PARAMS + ["yfeat_day", "ufeat_day"]
    for n in names:
        a = np.asarray(g.get_param(n), np.float64).ravel()
        b = np.asarray(o.get_param(n), np.float64).ravel()
        if a.size:
            assert np.max(np.abs(a - b) - 1e-5 * np.abs(b)) < 2e-5, n


@pytest.mark.parametrize("f", [0, 20, 33, 64, 96, 130, 190, 224, 256])
def test_user_stratum_at_the_edges_of_its_pairs_and_chunks(f):
    """Users with 1, 2, 3 ratings (a pair, a pair and a half), with a chunk of
    32 less and more one, and with a count past the ring of rows; the time-bin
    biases trained; every row layout."""
    counts = [1, 2, 3, 5, 6, 7, 8, 9, 31, 32, 33, 63, 64, 65, 97, 150]
    tr, pr = counted_sets(counts, 200, 3 + f)
    check_epochs(tr, pr, run_lm(f, 2, n_time_bins=48).replace(lr_tu=0.001, reset_u_epoch=2 if f == 64 else 1024))


def user_pass_ordinal(g, tr, cfg, u):
    """One user's ordinal-head pass over its training ratings, items frozen, in
    float64 (src/tsvdx4p.rs:535-613 with the head's gradient, src/lib.rs:562-598)."""
    P = {n: np.asarray(g.get_param(n), np.float64) for n in PARAMS + ["ycache", "ycache_bias", "tu_mean"]}
    th = np.array(cfg.ordinal_head.th_init)
    pu, p2, ub, al, cu = P["ufeat"][u], P["ufeat2"][u], P["ubias"][u], P["alpha_u"][u], P["cu"][u]
    but, bud = P["but_bin"][u].copy(), {}
    for t in np.nonzero(tr.user_idxs == u)[0]:
        i, day = tr.item_idxs[t], int(tr.dates[t])
        tb = min(day * cfg.n_time_bins // (int(tr.dates.max()) + 1), cfg.n_time_bins - 1)
        dt = day - P["tu_mean"][u]
        dv = np.sign(dt) * abs(dt) ** np.float64(np.float32(cfg.beta))
        qe = P["ifeat"][i] + P["ifeat_freq"][i * cfg.n_freq_bins]
        bi = P["ibias"][i] + P["bit_bin"][i, tb] + P["ibias_freq"][i, 0]
        x = (float(g.get_param("gbias")) + ub + but[tb] + al * dv + bud.get(day, 0.0) + P["ycache_bias"][u] + bi * cu
             + qe @ (pu + P["ycache"][u] + dv * p2))
        f = np.concatenate([[0.0], 1 / (1 + np.exp(-(th - x))), [1.0]])
        y = int(tr.raw_ratings[t])
        e = (f[y] * (1 - f[y]) - f[y - 1] * (1 - f[y - 1])) / max(f[y] - f[y - 1], 1e-6)
        ub, al = ub - cfg.lr_ub * e, al - cfg.lr_ta * e * dv
        but[tb] -= cfg.lr_tu * e
        bud[day] = bud.get(day, 0.0) - cfg.lr_ubd * e
        cu = cu - cfg.lr_cu * (e * bi + cfg.reg_cu * (cu - 1))
        pu, p2 = (pu - cfg.lr_u * (e * qe + cfg.reg_u * pu), p2 - cfg.lr_u2 * (e * qe * dv + cfg.reg_u2 * p2))
    return pu, p2, ub, al, cu, but


@pytest.mark.parametrize("f", [20, 64, 160])
def test_user_stratum_with_the_ordinal_head(f):
    """The head's gradient is not linear in the score: a pair's second rating
    must see the first one's update. A fold-in pass is the user stratum alone."""
    counts = [1, 2, 3, 31, 33, 64, 90]
    tr, pr = counted_sets(counts, 120, 9)
    cfg = run_lm(f, 1, n_time_bins=30).replace(
        lr_tu=0.001, sigma_u=0.1, sigma_i=0.1, ordinal_head=OrdinalHeadConfig((0.5, 1.25, 3.75, 5.5), 0.001, 0.0, 0.0))
    g = TxModel(tr, MaskedDataset(pr), cfg)
    g.rebuild_ycache()
    want = [user_pass_ordinal(g, tr, cfg, u) for u in range(len(counts))]
    foldin(g, np.arange(len(counts)), 1)
    for n, k in (("ufeat", 0), ("ufeat2", 1), ("ubias", 2), ("alpha_u", 3), ("cu", 4), ("but_bin", 5)):
        a = np.asarray(g.get_param(n), np.float64)
        assert np.max(np.abs(a - np.array([w[k] for w in want]))) < 2e-5, n


@pytest.mark.parametrize("f", [20, 64, 100, 160, 200, 256, 300])
def test_ycache_rebuild_is_bitwise_at_the_edges_of_its_row_groups(f):
    """The sums run over groups of 32, 16 or 8 rows, then four, then one, and a
    chunk of 32 items ahead; every add is in the reference's order."""
    counts = [1, 2, 3, 4, 5, 6, 7, 9, 13, 14, 15, 28, 29, 30, 31, 32, 45, 61, 62, 63, 94, 95]
    tr, pr = counted_sets(counts, 150, 17)
    cfg = run_lm(f, 1, n_time_bins=30)
    o, g = po.OracleModel(tr, MaskedDataset(pr), cfg), TxModel(tr, MaskedDataset(pr), cfg)
    yb = np.random.default_rng(5).normal(0, 0.1, tr.n_items).astype(np.float32)
    for m in (o, g):
        m.set_param("ybias", yb)
        m.rebuild_ycache()
    for n in ("ycache", "ycache_bias"):
        a = np.asarray(g.get_param(n), np.float32).ravel()
        assert np.array_equal(a.view(np.uint32), np.asarray(o.get_param(n), np.float32).ravel().view(np.uint32)), n


def counted_items(counts, n_users, seed):
    """Items with exactly these numbers of training ratings, users' ratings on
    few days so that several frequency bins meet in an item's rounds."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([rng.choice(n_users, size=n, replace=False) for n in counts])
    i = np.repeat(np.arange(len(counts)), counts)
    o = np.lexsort((i, u))
    u, i = u[o], i[o]
    d = 100 + 40 * (u % 7) + rng.integers(0, 1 + u % 5, size=len(u)) * 3
    tr = Dataset.from_ratings(u, i, rng.integers(1, 6, len(u)), d, n_users, len(counts), "items_tr")
    pu, pi = np.arange(n_users), np.full(n_users, len(counts) - 1)
    ok = ~np.isin(pu * len(counts) + pi, u * len(counts) + i)
    pr = Dataset.from_ratings(pu[ok], pi[ok], rng.integers(1, 6, ok.sum()), 100 + 40 * (pu[ok] % 7), n_users,
                              len(counts), "items_pr")
    return tr, pr


ITEM_COUNTS = [1, 2, 3, 5, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 96, 97, 128, 161]


@pytest.mark.parametrize("heavy", [1, 40, 100000])
@pytest.mark.parametrize("f", [0, 20, 40, 96, 128, 160, 224, 256])
def test_item_stratum_at_the_edges_of_its_rounds_and_pairs(f, heavy):
    """Items of one rating up to a few rounds of 32, all in rounds (heavy = 1),
    some, or all by one warp; strong item, bin and frequency updates and decays,
    so that a wrong weight inside a round shows."""
    tr, pr = counted_items(ITEM_COUNTS, 200, 5)
    cfg = run_lm(f, 2, n_time_bins=48).replace(lr_ti=0.002, lr_ibf=0.003, lr_iqf=0.004, reg_iqf=0.05, reg_i=0.05,
                                               sigma_u=0.1, sigma_i=0.1, sigma_iqf=0.1)
    check_epochs(tr, pr, cfg, heavy_item_ratings=heavy)


@pytest.mark.parametrize("f,bins", [(20, 64), (60, 12), (100, 16), (250, 64)])
def test_item_stratum_with_the_per_day_rows_and_many_bins(f, bins):
    """The per-day rows in the rounds' user rows; tables of up to 64 frequency
    bins beside the widest rows."""
    tr, pr = counted_items(ITEM_COUNTS, 200, 6)
    check_epochs(tr, pr, run_lm(f, 2, n_time_bins=30, low_memory=False).replace(n_freq_bins=bins, lr_iqf=0.004),
                 epochs=1)


def patterned_days(n_items, seed):
    """Users whose days follow patterns, in item order: each day once, days that
    come back one to four ratings later, runs of two and more (one over three
    chunks of 32), lone ratings beside runs; query pairs on every fourth day."""
    rng = np.random.default_rng(seed)
    u, i, d, pu, pi, pd = [], [], [], [], [], []
    patterns = ["abcdefgh", "ab", "abc", "abac", "abcd", "aab", "abb", "aabb", "abcca", "a" * 70 + "b"]
    k = 0
    for p in patterns:
        for n in (1, 2, 3, 31, 32, 33, 34, 65, 97):
            items = np.sort(rng.choice(n_items, size=n + 2, replace=False))
            q = rng.permutation(n + 2)
            days = [5 * k % 1400 + ord(p[j % len(p)]) + (3 * j if p == "abcdefgh" else 0) for j in range(n)]
            u += [k] * n
            i += list(items[np.sort(q[:n])])
            d += days
            if k % 4 == 0:
                pu += [k] * 2
                pi += list(items[q[n:]])
                pd += [days[0], days[-1]]
            k += 1
    tr = Dataset.from_ratings(u, i, rng.integers(1, 6, len(u)), d, k, n_items, "days_tr")
    o = np.lexsort((np.array(pu), np.array(pi)))
    pr = Dataset.from_ratings(np.array(pu)[o], np.array(pi)[o], rng.integers(1, 6, len(pu)), np.array(pd)[o], k,
                              n_items, "days_pr")
    return tr, pr


@pytest.mark.parametrize("f,full_su,lr_ud", [(20, True, 0.005), (60, True, 0.005), (60, False, 0.005), (60, True, 0.0),
                                             (90, True, 0.005), (128, True, 0.005), (190, True, 0.005),
                                             (256, True, 0.005)])
def test_user_stratum_with_the_per_day_rows(f, full_su, lr_ud):
    """Pairs of lone ratings, ufeat_day rows handed on between ratings of one day,
    and runs of equal dates; two epochs, so that the day rows are not zero."""
    tr, pr = patterned_days(150, 7)
    check_epochs(tr, pr, run_lm(f, 2, n_time_bins=30, low_memory=False).replace(full_su=full_su, lr_ud=lr_ud))


@pytest.mark.parametrize("f,bins", [(257, 16), (600, 16), (1000, 16), (1100, 16), (1600, 30), (2048, 16), (2100, 16)])
def test_rows_above_256_columns(f, bins):
    """A block per unit up to 2,048 columns, with the q^f rows in shared memory (16 or
    8 ratings in the ring) and in the table; a warp per unit above."""
    counts = [1, 2, 3, 6, 7, 8, 15, 16, 17, 31, 32, 33, 34, 46, 63, 64, 65, 97, 1, 2]
    tr, pr = counted_sets(counts, 120, 8)
    check_epochs(tr, pr, run_lm(f, 2, n_time_bins=30).replace(n_freq_bins=bins, lr_iqf=0.004), epochs=1)
    tr, pr = counted_items([c for c in ITEM_COUNTS if c <= 150], 150, 9)
    check_epochs(tr, pr, run_lm(f, 2, n_time_bins=30).replace(n_freq_bins=bins, lr_iqf=0.004), epochs=1)


@pytest.mark.parametrize("f,low_memory", [(20, True), (60, False), (96, True), (256, True), (256, False), (400, True)])
def test_many_rows_score_as_few(f, low_memory):
    """Predictions by groups of 2 to 32 rows a warp are, bit for bit, those of a warp
    per row, rows outside the tables (NaN) among them; the RMSE is that of these
    scores (sums of n squares in FP64: relative error below n 2^-53 = 4e-11)."""
    tr, pr = counted_items(ITEM_COUNTS, 200, 10)
    g = TxModel(tr, MaskedDataset(pr), run_lm(f, 1, n_time_bins=30, low_memory=low_memory))
    g.fit_epoch(tr, pr, 1)
    rng = np.random.default_rng(11)
    n = 303150
    u, i = rng.integers(0, 200, n), np.sort(rng.integers(0, len(ITEM_COUNTS), n))
    d = rng.choice(np.concatenate([tr.dates, rng.integers(0, 2000, 50)]), n)

    def scores(sel, v):
        t = [torch.as_tensor(np.ascontiguousarray(x[sel]), device="cuda", dtype=ty)
             for x, ty in ((v, torch.int32), (i, torch.int32), (d, torch.int16))]
        out = torch.empty(len(t[0]), device="cuda")
        torch.cuda.synchronize()
        g._check(g._L.tsvd_predict_batch_device(g.h, *[C.c_void_p(x.data_ptr()) for x in t], len(out),
                                                C.c_void_p(out.data_ptr())))
        torch.cuda.synchronize()
        return out.cpu().numpy().view(np.uint32)

    wild = u.copy()
    wild[rng.integers(0, n, 3000)] = 200
    wild[rng.integers(0, n, 3000)] = -1
    few = np.concatenate([scores(slice(a, a + 15000), wild) for a in range(0, n, 15000)])
    assert np.isnan(few.view(np.float32)).sum() > 5000
    for m in (18943, 18944, 18977, 75777, n):
        assert np.array_equal(scores(slice(0, m), wild), few[:m]), m
    raw = rng.integers(1, 6, n)
    o = np.lexsort((u, i))
    u, i, d = u[o], i[o], d[o]
    held = Dataset.from_ratings(u, i, raw, d, 200, len(ITEM_COUNTS), "held")
    e = (scores(slice(0, n), u).view(np.float32) - held.residuals.astype(np.float32)).astype(np.float64)
    want = np.sqrt(np.mean(e * e))
    assert abs(g.calc_rmse(held) - want) < 1e-10 * want
