"""The work that a user of this framework has it do, as cases of one call each.

A case is a dict of plain values; `listed()` gives the named ones, `draw(rng)`
more of the same ranges. `prepare(case, seed)` makes what a program holds
before the call (the data set, a model with trained-looking parameters, row
arrays), `run(state)` is one pass through the public entry points and returns
its results whole, `work(case)` the bytes and operations the pass cannot do
without, and `exact(case, seed)` the same results from plain torch in 64 bits.

Kinds of case:
  epoch    one training epoch of a TxModel (stratified, the default schedule):
           Regressor::fit_epoch, the call a training job makes n_epochs times
  group    one epoch of several variants over one data set (TxGroup)
  predict  predictions of device-resident rows (probe and qualifying set)
  rows     predictions and held-out RMSE of rows in host buffers
  foldin   user-side passes over new users with the item tables frozen
  encoder  one epoch of the learned warm start's encoder

Data are seeded stand-ins of the Netflix Prize set's shape: Zipf-popular items,
lognormal user activity, ratings on session days, a held-out and query set.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from netflix_prize_b200.abi import PREC_BF16_READ, PREC_FP32
from netflix_prize_b200.config import OrdinalHeadConfig, TxConfig
from netflix_prize_b200.data import Dataset, MaskedDataset
from netflix_prize_b200.encoder import UserEncoder, foldin
from netflix_prize_b200.model import TxGroup, TxModel

N_DAYS = 2243  # days 0..2242 of the Netflix Prize set


def _case(kind, users, items, ratings, f, **more):
    c = dict(kind=kind, users=users, items=items, ratings=ratings, f=f, time_bins=29, freq_bins=16, per_day=False,
             ordinal=False, bf16=False, rows=0, passes=0, batch=0, variants=0)
    c.update(more)
    return c


def listed():
    n = lambda name, c: dict(c, name=name)
    return [
        # the headline workload: an epoch over the whole Netflix-shaped set at f = 256
        n("netflix f256", _case("epoch", 480_189, 17_770, 100_480_507, 256, time_bins=30)),
        # a quarter of the set with the read tables as BF16 copies (the precision form)
        n("25M f64 bf16", _case("epoch", 120_000, 17_770, 25_000_000, 64, time_bins=30, bf16=True)),
        # a development set: the size on which configurations are tried out
        n("1M f32", _case("epoch", 10_000, 2_000, 1_000_000, 32, time_bins=30)),
        # the smallest set that is trained on in tests and smoke runs
        n("20k f16", _case("epoch", 500, 200, 20_000, 16, time_bins=30)),
        # tsvdx4-60: 60 columns with the per-day terms
        n("6M f60 per-day", _case("epoch", 30_000, 8_000, 6_000_000, 60, per_day=True)),
        # tsvdx4-s20fo: the ordinal head, 24 frequency bins
        n("3M f20 ordinal", _case("epoch", 15_003, 4_001, 3_000_000, 20, time_bins=25, freq_bins=24, ordinal=True)),
        # tsvdx4-400lm: rows above 256 columns
        n("2M f400", _case("epoch", 10_007, 3_001, 2_000_000, 400)),
        # a hyperparameter search: four factor sizes trained together
        n("4 variants 1M", _case("group", 10_000, 2_000, 1_000_000, 128, time_bins=30, variants=4)),
        # predictions of the probe and qualifying sets (4.2 M rows) after a Netflix-sized training
        n("predict 4.2M f256", _case("predict", 480_189, 17_770, 20_000_000, 256, rows=4_225_526)),
        # a small scoring call: host rows in, predictions and RMSE out
        n("rows 1000 f64", _case("rows", 10_000, 2_000, 1_000_000, 64, rows=1_000)),
        # new users folded into a trained model
        n("foldin 8k f128", _case("foldin", 40_000, 17_770, 8_000_000, 128, rows=8_001, passes=3)),
        # the warm-start encoder's training epoch
        n("encoder 10k f32", _case("encoder", 10_000, 2_000, 1_000_000, 32, rows=10_000, batch=512)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["epoch", "group", "predict", "rows", "foldin", "encoder"], [10, 1, 2, 2, 2, 1])[0]
    ratings = _log_int(rng, 20_000, 25_000_000)
    f = min(256, _log_int(rng, 1, 300))
    more = dict(time_bins=rng.choice([20, 25, 29, 30, 48]), freq_bins=rng.choice([12, 16, 16, 24]))
    if kind == "epoch":
        form = rng.choices(["plain", "bf16", "per_day", "ordinal", "wide"], [5, 1, 2, 1, 1])[0]
        if form == "bf16":
            more["bf16"] = True
        elif form == "per_day":
            ratings, f = min(ratings, 6_000_000), min(f, 160)
            more.update(per_day=True, ordinal=rng.random() < 0.5)
        elif form == "ordinal":
            ratings = min(ratings, 6_000_000)
            more["ordinal"] = True
        elif form == "wide":
            ratings, f = min(ratings, 2_000_000), _log_int(rng, 257, 700)
    elif kind == "group":
        ratings = min(ratings, 2_000_000)
        more["variants"] = rng.randint(2, 4)
    elif kind == "predict":
        ratings = min(ratings, 10_000_000)
        more.update(rows=_log_int(rng, 50_000, 4_000_000), per_day=f <= 96 and rng.random() < 0.25)
    elif kind == "rows":
        ratings = min(ratings, 2_000_000)
        more["rows"] = _log_int(rng, 1, 200_000)
    elif kind == "foldin":
        ratings, f = min(ratings, 8_000_000), max(f, 1)
        more["passes"] = rng.randint(1, 4)
    elif kind == "encoder":
        ratings, f = min(ratings, 1_000_000), max(f, 4)
        more["batch"] = rng.choice([100, 256, 512, 1024])
    per_user = rng.uniform(60, 260)
    users = max(64, int(ratings / per_user))
    items = max(_log_int(rng, 200, 17_770), int(per_user * 3))
    if kind in ("foldin", "encoder"):
        more["rows"] = rng.randint(max(1, users // 20), users if kind == "encoder" else max(2, users // 4))
    return _case(kind, users, items, ratings, f, **more)


# ---------------------------------------------------------------------------
# data
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, salt):
    return torch.Generator(_device()).manual_seed((seed * 1_000_003 + salt) & 0x7FFFFFFF)


def _columns(case, seed):
    """The data set's columns on the device: training rows sorted by (user,
    item), pr rows by (item, user). Each (user, item) pair is rated with
    probability min(1, c_u w_i), c_u set by the user's activity."""
    U, I, dev = case["users"], case["items"], _device()
    g = _gen(seed, 1)
    act = torch.exp(1.25 * torch.randn(U, generator=g, device=dev, dtype=torch.float64))
    want = (act * (case["ratings"] / act.sum())).clamp(2.0, 0.9 * I)
    want = (want * (case["ratings"] / want.sum())).clamp(1.0, 0.9 * I)
    rank_item = torch.randperm(I, generator=g, device=dev)
    w = torch.arange(1, I + 1, device=dev, dtype=torch.float64) ** -1.05
    w = w / w.sum()
    tail = torch.cat([w.flip(0).cumsum(0).flip(0), torch.zeros(1, device=dev, dtype=torch.float64)])
    lo, hi = torch.zeros(U, device=dev, dtype=torch.float64), torch.full((U,), 60.0, device=dev, dtype=torch.float64)
    for _ in range(50):  # log c_u
        mid = 0.5 * (lo + hi)
        c = torch.exp(mid)
        m = I - torch.searchsorted(w.flip(0).contiguous(), 1.0 / c)  # items with c w >= 1
        ok = m + c * tail[m] < want
        lo, hi = torch.where(ok, mid, lo), torch.where(ok, hi, mid)
    w_item = torch.empty(I, device=dev)
    w_item[rank_item] = w.float()
    c = torch.exp(hi).float()
    top = int(rank_item[0])
    rows = max(1, (1 << 26) // I)
    parts = []
    for a in range(0, U, rows):
        p = c[a:a + rows, None] * w_item
        hit = torch.rand(p.shape, generator=g, device=dev) < p
        hit[:, top] |= ~hit.any(1)  # nobody without a rating
        parts.append((hit.nonzero() + torch.tensor([a, 0], device=dev)).to(torch.int32))
    pair = torch.cat(parts)
    del parts
    u, i = pair[:, 0].contiguous(), pair[:, 1].contiguous()
    del pair
    cnt = torch.bincount(u, minlength=U)
    start = torch.randint(0, N_DAYS - 1, (U,), generator=g, device=dev)
    span = (torch.rand(U, generator=g, device=dev) * 700).long().clamp(min=1)
    span = torch.minimum(span, N_DAYS - 1 - start)
    sess = (cnt.double() ** 0.55 * 1.2).long().clamp(min=1)
    bu = 0.4 * torch.randn(U, generator=g, device=dev)
    bi = 0.5 * torch.randn(I, generator=g, device=dev)
    pu = 0.5 * torch.randn((U, 4), generator=g, device=dev)
    qi = 0.5 * torch.randn((I, 4), generator=g, device=dev)

    def day_of(uu, k):  # session k of a user
        return start[uu] + ((uu * 40503 + k * 7919) % 65521) % (span[uu] + 1)

    def rate(uu, ii):
        s = 3.6 + bu[uu] + bi[ii] + (pu[uu] * qi[ii]).sum(1) + 0.9 * torch.randn(len(uu), generator=g, device=dev)
        return s.round().clamp(1, 5).to(torch.int8)

    day, raw = torch.empty(len(u), device=dev, dtype=torch.int16), torch.empty(len(u), device=dev, dtype=torch.int8)
    for a in range(0, len(u), 1 << 24):
        uu, ii = u[a:a + (1 << 24)].long(), i[a:a + (1 << 24)].long()
        k = (torch.rand(len(uu), generator=g, device=dev) * sess[uu]).long()
        day[a:a + len(uu)] = day_of(uu, k).to(torch.int16)
        raw[a:a + len(uu)] = rate(uu, ii)
    # pr: about nine popular unrated items a user, a third of them held-out ratings
    qu = torch.arange(U, device=dev).repeat_interleave(10)
    r = torch.rand(len(qu), generator=g, device=dev, dtype=torch.float64)
    qv = rank_item[torch.searchsorted(w.cumsum(0), r).clamp(max=I - 1)]
    key = torch.unique(qu * I + qv)
    off = torch.cat([torch.zeros(1, device=dev, dtype=torch.long), cnt.cumsum(0)])
    rated = torch.zeros(len(key), device=dev, dtype=torch.bool)
    a0, a1 = off[key // I].clone(), off[key // I + 1].clone()
    end, it = a1.clone(), (key % I).to(torch.int32)
    for _ in range(16):  # the pair's place among the user's items
        mid = (a0 + a1) // 2
        less = (a0 < a1) & (i[mid.clamp(max=len(i) - 1)] < it)
        a0, a1 = torch.where(less, mid + 1, a0), torch.where(less | (a0 >= a1), a1, mid)
    rated = (a0 < end) & (i[a0.clamp(max=len(i) - 1)] == it)
    key = key[~rated]
    key = key[torch.argsort((key % I) * U + key // I)]
    vu, vi = key // I, key % I
    vday = (start[vu] + span[vu] + torch.randint(0, 60, (len(vu),), generator=g, device=dev)).clamp(max=N_DAYS - 1)
    same = torch.rand(len(vu), generator=g, device=dev) < 0.3  # some on a day with training ratings
    vday = torch.where(same, day_of(vu, (torch.rand(len(vu), generator=g, device=dev) * sess[vu]).long()), vday)
    test = (torch.rand(len(vu), generator=g, device=dev) < 2.0 / 3.0).to(torch.int8)
    vraw = torch.where(test != 0, torch.zeros_like(test), rate(vu, vi))
    return dict(u=u, i=i, day=day, raw=raw), dict(u=vu.int(), i=vi.int(), day=vday.to(torch.int16), raw=vraw, test=test)


def _sets(case, cols):
    t, v = ({k: x.cpu().numpy() for k, x in d.items()} for d in cols)
    U, I = case["users"], case["items"]
    tr = Dataset.from_ratings(t["u"], t["i"], t["raw"], t["day"], U, I, "train")
    pr = Dataset.from_ratings(v["u"], v["i"], v["raw"], v["day"], U, I, "pr", is_test=v["test"])
    return tr, pr


def _config(case, variant=0, seed=42):
    over = {}
    if variant:  # a search over factor sizes and learning rates
        over = dict(lr_u=0.003 + 0.001 * variant, lr_i=0.0036 + 0.001 * variant)
    if case["ordinal"]:  # the small_o presets' rates
        over = dict(lr_u=0.003, lr_ud=0.0015, lr_u2=1e-5, lr_ub=0.006, lr_ubd=0.006, lr_i=0.0072, lr_ib=0.0072,
                    lr_y=0.0012, lr_yb=2e-6, lr_ti=0.0001, lr_ta=1.5e-5, reg_u=0.04, reg_i=0.007, reg_yd=0.04,
                    reset_u_epoch=1024, ordinal_head=OrdinalHeadConfig((0.5, 1.25, 3.75, 5.5), 0.001, 0.0, 0.0))
    return TxConfig(n_feat=_widths(case)[variant], n_epochs=20, seed=seed, n_time_bins=case["time_bins"],
                    n_freq_bins=case["freq_bins"], low_memory=not case["per_day"], **over)


def _widths(case):
    if case["kind"] != "group":
        return [case["f"]]
    return [max(1, case["f"] >> k) for k in range(case["variants"])]


# ---------------------------------------------------------------------------
# parameters: a model some epochs into its training
# ---------------------------------------------------------------------------
def _tables(case, n_ud, f):
    """(name, rows, columns, scale, offset) of the trained tables."""
    U, I, T, NF = case["users"], case["items"], case["time_bins"], case["freq_bins"]
    z = 0.4 / max(f, 1) ** 0.25
    t = [("ufeat", U, f, z, 0), ("ufeat2", U, f, 0.01 * z, 0), ("ifeat", I, f, z, 0), ("yfeat", I, f, 0.2 * z, 0),
         ("ifeat_freq", I * NF, f, 0.05 * z, 0), ("ubias", U, 1, 0.3, 0), ("ibias", I, 1, 0.3, 0),
         ("alpha_u", U, 1, 0.01, 0), ("but_bin", U, T, 0.05, 0), ("bit_bin", I, T, 0.05, 0), ("ybias", I, 1, 0.01, 0),
         ("ibias_freq", I, NF, 0.02, 0), ("cu", U, 1, 0.05, 1), ("ubias_day", n_ud, 1, 0.1, 0)]
    if case["per_day"]:
        t += [("yfeat_day", I, f, 0.1 * z, 0), ("ufeat_day", n_ud, f, 0.1 * z, 0)]
    return [x for x in t if x[2] > 0]


def _values(seed, k, rows, cols, scale, offset):
    g = _gen(seed, 100 + k)
    return torch.randn((rows, cols), generator=g, device=_device()).mul_(scale).add_(offset)


def _n_ud(model, case):
    a, b = C.c_uint64(), C.c_uint64()
    model._check(model._L.tsvd_user_day_range(model.h, 0, case["users"], C.byref(a), C.byref(b)))
    return b.value


def _rows(model, name, rows, tensor, to_model):
    model._check(model._L.tsvd_copy_rows(model.h, name.encode(), 0, rows, C.c_void_p(tensor.data_ptr()), to_model))


def _load(model, case, seed, f):
    tables = _tables(case, _n_ud(model, case), f)
    for k, (name, rows, cols, scale, offset) in enumerate(tables):
        v = _values(seed, k, rows, cols, scale, offset)
        torch.cuda.synchronize()
        _rows(model, name, rows, v, 1)
    return [(name, rows, cols) for name, rows, cols, _, _ in tables]


def _take(model, tables, buffers):
    """The tables as packed device tensors, in the program's own buffers."""
    for name, rows, _ in tables:
        _rows(model, name, rows, buffers[name], 0)
    return buffers


def _buffers(case, tables):
    """One buffer a table; those of (user, day) rows, whose number is the data's, with room for any."""
    most = _most_ud(case)
    n = lambda name, rows: most if name in ("ubias_day", "ufeat_day") else rows
    return {name: torch.zeros((n(name, rows), cols), device="cuda") for name, rows, cols in tables}


def _most_ud(case):
    U = case["users"]
    return int(U * (1.2 * (1.1 * case["ratings"] / U) ** 0.55 + 11))


USER_TABLES = ("ufeat", "ufeat2", "ubias", "alpha_u", "cu", "but_bin", "ubias_day")


def _query(case, seed):
    """Rows to predict: pairs sorted by (item, user) as the pr set is, dates over the whole range."""
    g = _gen(seed, 3)
    n, dev = case["rows"], _device()
    u = torch.randint(0, case["users"], (n,), generator=g, device=dev)
    i = (torch.rand(n, generator=g, device=dev) ** 3 * case["items"]).long().clamp(max=case["items"] - 1)
    o = torch.argsort(i * case["users"] + u)
    day = torch.randint(0, N_DAYS, (n,), generator=g, device=dev)
    return u[o].int(), i[o].int(), day.to(torch.int16)


def _some_users(case, seed):
    g = _gen(seed, 4)
    return torch.randperm(case["users"], generator=g, device=_device())[:case["rows"]].cpu().numpy().astype(np.uint32)


ENC = ["e_item", "e_rate", "e_date", "w1", "b1", "w2", "b2", "w3", "b3"]


def _enc_values(case, seed):
    O, hid, emb = case["f"] + 2, 512, 128
    shape = [(case["items"] * 5, emb), (5, emb), (case["time_bins"], emb), (emb, hid), (hid, 1), (hid, hid), (hid, 1),
             (hid, O), (O, 1)]
    scale = [0.05, 0.05, 0.05, emb ** -0.5, 0.05, hid ** -0.5, 0.05, hid ** -0.5, 0.05]
    return {n: _values(seed, 50 + k, s[0], s[1], x, 0) for k, (n, s, x) in enumerate(zip(ENC, shape, scale))}


def prepare(case, seed):
    cols = _columns(case, seed)
    tr, pr = _sets(case, cols)
    del cols
    s = {"kind": case["kind"], "epoch": 0}
    if case["kind"] == "group":
        cfgs = [_config(case, k) for k in range(case["variants"])]
        g = TxGroup(tr, MaskedDataset(pr), cfgs)
        s["group"] = g
        s["tables"] = [_load(m, case, seed + k, f) for k, (m, f) in enumerate(zip(g.models, _widths(case)))]
        s["buffers"] = [_buffers(case, t) for t in s["tables"]]
        torch.cuda.empty_cache()
        return s
    prec = PREC_BF16_READ if case["bf16"] else PREC_FP32
    m = TxModel(tr, MaskedDataset(pr), _config(case), precision=prec)
    s["model"], s["tables"] = m, _load(m, case, seed, case["f"])
    if case["kind"] == "foldin":
        s["tables"] = [t for t in s["tables"] if t[0] in USER_TABLES]
    if case["kind"] in ("epoch", "foldin"):
        s["buffers"] = _buffers(case, s["tables"])
    if case["kind"] in ("predict", "rows", "foldin"):
        m.rebuild_ycache()
    if case["kind"] == "predict":
        s["u"], s["i"], s["day"] = _query(case, seed)
        s["out"] = torch.empty(case["rows"], device="cuda")
        s["ptr"] = [C.c_void_p(s[k].data_ptr()) for k in ("u", "i", "day")]
    elif case["kind"] == "rows":
        u, i, d = (x.cpu().numpy() for x in _query(case, seed))
        raw = (1 + (u * 7 + i * 13) % 5).astype(np.int8)
        s["held"] = Dataset.from_ratings(u, i, raw, d, case["users"], case["items"], "held")
    elif case["kind"] == "foldin":
        s["users"], s["passes"] = _some_users(case, seed), case["passes"]
    elif case["kind"] == "encoder":
        s["users"], s["batch"] = _some_users(case, seed), case["batch"]
        s["enc"] = UserEncoder(m, tr.raw_ratings, s["users"], seed=5, lr=1e-4)
        for n, v in _enc_values(case, seed).items():
            s["enc"].set(n, v.cpu().numpy())
    torch.cuda.empty_cache()
    return s


def run(s):
    kind = s["kind"]
    if kind == "epoch":
        s["epoch"] = s["epoch"] % 20 + 1
        s["model"].fit_epoch(epoch=s["epoch"])
        return _take(s["model"], s["tables"], s["buffers"])
    if kind == "group":
        s["epoch"] = s["epoch"] % 20 + 1
        s["group"].fit_epoch(s["epoch"])
        return [_take(m, t, b) for m, t, b in zip(s["group"].models, s["tables"], s["buffers"])]
    if kind == "predict":
        m = s["model"]
        m._check(m._L.tsvd_predict_batch_device(m.h, *s["ptr"], len(s["out"]), C.c_void_p(s["out"].data_ptr())))
        return s["out"]
    if kind == "rows":
        h = s["held"]
        return {"pred": s["model"].predict_batch(h.user_idxs, h.item_idxs, h.dates), "rmse": s["model"].calc_rmse(h)}
    if kind == "foldin":
        foldin(s["model"], s["users"], s["passes"])
        return _take(s["model"], s["tables"], s["buffers"])
    loss = s["enc"].train_epoch(s["users"], batch=s["batch"])
    return {"loss": loss, **{n: s["enc"].get(n) for n in ENC}}


def work(case):
    U, I, R, T, NF = case["users"], case["items"], case["ratings"], case["time_bins"], case["freq_bins"]
    n_ud = 0.2 * R  # (user, day) pairs, about
    by, fl = 0.0, 0.0
    for f in _widths(case):
        user, item = 4.0 * U * (2 * f + T + 3), 4.0 * I * (2 * f + NF * f + T + NF + 2)
        day = 4.0 * n_ud * (1 + (f if case["per_day"] else 0))
        if case["kind"] in ("epoch", "group"):
            # ratings (item, residual, date) read once, every table read and written once; per rating a dot, the
            # updates of the rows it meets in either stratum, and its part of the NSVD1 sums
            by += 10.0 * R + 2 * (user + item + day)
            fl += R * f * (36.0 if case["per_day"] else 32.0)
        elif case["kind"] in ("predict", "rows"):
            n = case["rows"]
            by += min(user + 4.0 * U * f, 4.0 * n * (3 * f + 5)) + min(item, 4.0 * n * (2 * f + 3)) + 14.0 * n
            fl += 8.0 * n * f
        elif case["kind"] == "foldin":
            n = case["rows"] / U
            by += 10.0 * R * n + 2 * (user + day) * n + min(item, 4.0 * R * n * f) + 4.0 * U * n * f
            fl += case["passes"] * R * n * f * 16.0
        else:
            n, steps = case["rows"], math.ceil(case["rows"] / case["batch"])
            w = 128 * 512 + 512 * 512 + 512 * (f + 2)
            by += 6.0 * R * n / U + steps * 28.0 * (I * 5 * 128 + w)
            fl += 6.0 * n * w + 4.0 * 128 * R * n / U
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """The data set's derived columns and the model's tables in float64."""

    def __init__(self, case, seed, cols, variant=0):
        t, v = cols
        self.c = c = _config(case, variant)
        self.case, dev = case, _device()
        U, I, NF = case["users"], case["items"], case["freq_bins"]
        self.u, self.i, day = t["u"].long(), t["i"].long(), t["day"].long()
        self.vu, self.vi, vday = v["u"].long(), v["i"].long(), v["day"].long()
        self.n, self.cnt = len(self.u), torch.bincount(self.u, minlength=U)
        self.vcnt = torch.bincount(self.vu, minlength=U)
        self.off = torch.cat([self.cnt.new_zeros(1), self.cnt.cumsum(0)])
        self.day_range = int(day.max()) + 1
        mean = torch.zeros(U, device=dev, dtype=torch.float64).index_add_(0, self.u, day.double())
        for x in torch.nonzero(mean >= 2.0 ** 24)[:, 0].tolist():  # the mean day is a sum of 32-bit floats
            d = day[int(self.off[x]):int(self.off[x + 1])].cpu().numpy().astype(np.float32)
            mean[x] = float(np.add.accumulate(d, dtype=np.float32)[-1])
        self.mean = (mean / self.cnt.clamp(min=1)).float().double()
        self.ud_key, inv = torch.unique(torch.cat([self.u * 4096 + day, self.vu * 4096 + vday]), return_inverse=True)
        self.ud, self.vud = inv[:self.n], inv[self.n:]
        n_day = torch.bincount(inv)
        cap = sum((n_day >= 2 ** k).long() for k in range(1, NF)).clamp(max=NF - 1)  # floor(log2(ratings of the day))
        self.bin_of_ud, self.fb = cap, cap[self.ud]
        self.dev, self.tb = self.dev_of(self.u, day), self.tbin(day)
        res = t["raw"].double()
        self.res, self.gbias = res, float(np.float32((res.sum() / self.n).item()))
        # runs of equal dates within a user
        new = torch.ones(self.n, device=dev, dtype=torch.bool)
        new[1:] = (self.u[1:] != self.u[:-1]) | (day[1:] != day[:-1])
        self.run = new.long().cumsum(0) - 1
        self.p = {}
        for k, (name, rows, k_cols, scale, offset) in enumerate(
                _tables(case, len(self.ud_key), _widths(case)[variant])):
            self.p[name] = _values(seed, k, rows, k_cols, scale, offset).double()
        f = _widths(case)[variant]
        for name, rows in (("ufeat", U), ("ufeat2", U), ("ifeat", I), ("yfeat", I), ("ifeat_freq", I * NF),
                           ("yfeat_day", I), ("ufeat_day", len(self.ud_key))):
            if name not in self.p and (not name.endswith("_day") or case["per_day"]):
                self.p[name] = torch.zeros((rows, f), device=dev, dtype=torch.float64)
        self.names = [x[0] for x in _tables(case, len(self.ud_key), f)]

    def out(self, names=None):
        """The tables in run()'s layout."""
        got, most = {}, _most_ud(self.case)
        for n in self.names:
            if names is None or n in names:
                v = self.p[n]
                if n in ("ubias_day", "ufeat_day"):
                    v = torch.cat([v, v.new_zeros((most - len(v), v.shape[1]))])
                got[n] = v
        return got

    def tbin(self, day):
        return (day * self.c.n_time_bins // self.day_range).clamp(max=self.c.n_time_bins - 1)

    def dev_of(self, u, day):
        d = day.double() - self.mean[u]
        return torch.sign(d) * d.abs() ** float(np.float32(self.c.beta))

    def lr(self, name):
        return float(np.float32(getattr(self.c, name)))

    def err(self, score, res):
        if self.c.ordinal_head is None:
            return score - res
        th = torch.tensor(self.c.ordinal_head.th_init, device=score.device, dtype=torch.float64)
        f = torch.zeros((len(score), 6), device=score.device, dtype=torch.float64)
        f[:, 5] = 1.0
        f[:, 1:5] = torch.sigmoid(th[None, :] - score[:, None])
        a = f * (1 - f)
        y = res.long()[:, None]
        get = lambda x, k: x.gather(1, k)[:, 0]
        return (get(a, y) - get(a, y - 1)) / (get(f, y) - get(f, y - 1)).clamp(min=1e-6)

    def cache(self):
        p = self.p
        sq = torch.sqrt((self.cnt + self.vcnt).clamp(min=1).double())[:, None]
        for name, out in (("yfeat", "ycache"), ("ybias", "ycache_bias")):
            y = p[name]
            acc = torch.zeros((len(self.cnt), y.shape[1]), device=y.device, dtype=torch.float64)
            for key, item in ((self.u, self.i), (self.vu, self.vi)):
                for a in range(0, len(key), 1 << 20):
                    acc.index_add_(0, key[a:a + (1 << 20)], y[item[a:a + (1 << 20)]])
            p[out] = acc / sq
        if self.case["per_day"]:
            y = p["yfeat_day"]
            acc = torch.zeros((len(self.ud_key), y.shape[1]), device=y.device, dtype=torch.float64)
            n = torch.zeros(len(self.ud_key), device=y.device, dtype=torch.float64)
            for key, item in ((self.ud, self.i), (self.vud, self.vi)):
                acc.index_add_(0, key, y[item])
                n.index_add_(0, key, torch.ones(len(key), device=y.device, dtype=torch.float64))
            p["ycache_day"] = acc / torch.sqrt(n)[:, None]

    def users_pass(self, users):
        """The user stratum over `users`; their NSVD1 gradients in self.g, self.ge."""
        p, c, day = self.p, self.c, self.case["per_day"]
        lr, NF = self.lr, c.n_freq_bins
        users = users[torch.argsort(self.cnt[users], descending=True)]
        steps = self.cnt[users].cpu().numpy()
        U, F = len(self.cnt), p["ufeat"].shape[1]
        self.g = torch.zeros((U, F), device=users.device, dtype=torch.float64)
        self.ge = torch.zeros(U, device=users.device, dtype=torch.float64)
        if day:
            n_runs = int(self.run[-1]) + 1
            self.seqd = torch.zeros((n_runs, F), device=users.device, dtype=torch.float64)
            sud = torch.zeros_like(self.seqd).index_add_(0, self.run, p["yfeat_day"][self.i])
            nd = torch.bincount(self.run, minlength=n_runs).double()
            ud_of_run = torch.zeros(n_runs, device=users.device, dtype=torch.long)
            ud_of_run[self.run] = self.ud
            pr_sum = torch.zeros_like(p["ufeat_day"]).index_add_(0, self.vud, p["yfeat_day"][self.vi])
            pr_n = torch.bincount(self.vud, minlength=len(self.ud_key)).double()
            self.nd = torch.sqrt(nd + pr_n[ud_of_run])
            sud = (sud + pr_sum[ud_of_run]) / self.nd[:, None]
        for k in range(int(steps[0]) if len(steps) else 0):
            m = int(np.searchsorted(-steps, -k, side="left"))
            u = users[:m]
            t = self.off[u] + k
            i, tb, ud, dv = self.i[t], self.tb[t], self.ud[t], self.dev[t]
            fb = self.fb[t] if day else torch.zeros_like(i)
            qe = p["ifeat"][i] + p["ifeat_freq"][i * NF + fb]
            bi = p["ibias"][i, 0] + p["bit_bin"][i, tb] + p["ibias_freq"][i, fb]
            pu, p2, cu = p["ufeat"][u], p["ufeat2"][u], p["cu"][u, 0]
            pe = pu + p["ycache"][u] + dv[:, None] * p2
            if day:
                pud = p["ufeat_day"][ud]
                pe = pe + pud + sud[self.run[t]]
            score = (self.gbias + p["ubias"][u, 0] + p["but_bin"][u, tb] + p["alpha_u"][u, 0] * dv
                     + p["ubias_day"][ud, 0] + p["ycache_bias"][u, 0] + bi * cu + (qe * pe).sum(1))
            e = self.err(score, self.res[t])
            eq = e[:, None] * qe
            p["ubias"][u, 0] -= lr("lr_ub") * e
            p["but_bin"][u, tb] -= lr("lr_tu") * e
            p["alpha_u"][u, 0] -= lr("lr_ta") * e * dv
            p["ubias_day"][ud, 0] -= lr("lr_ubd") * e
            p["cu"][u, 0] -= lr("lr_cu") * (e * bi + lr("reg_cu") * (cu - 1))
            self.ge[u] += e
            self.g[u] += eq
            p["ufeat"][u] -= lr("lr_u") * (eq + lr("reg_u") * pu)
            p["ufeat2"][u] -= lr("lr_u2") * (eq * dv[:, None] + lr("reg_u2") * p2)
            if day:
                self.seqd[self.run[t]] += eq
                p["ufeat_day"][ud] -= lr("lr_ud") * (eq + lr("reg_ud") * pud)
        norm = torch.sqrt((self.cnt + self.vcnt).clamp(min=1).double())
        self.g /= norm[:, None]
        self.ge /= norm

    def epoch(self):
        p, c, lr, day = self.p, self.c, self.lr, self.case["per_day"]
        I, NF = self.case["items"], c.n_freq_bins
        dev = self.u.device
        self.cache()
        self.users_pass(torch.nonzero(self.cnt > 0)[:, 0])
        nc = torch.bincount(self.i, minlength=I).double().clamp(min=1)[:, None]
        rated = (torch.bincount(self.i, minlength=I) > 0).double()[:, None]

        def sums(values, key):  # the mean over each item's ratings of their users' (or runs') rows
            acc = torch.zeros((I, values.shape[1]), device=dev, dtype=torch.float64)
            for a in range(0, self.n, 1 << 20):
                acc.index_add_(0, self.i[a:a + (1 << 20)], values[key[a:a + (1 << 20)]])
            return acc / nc

        p["yfeat"] -= rated * lr("lr_y") * (sums(self.g, self.u) + lr("reg_y") * p["yfeat"])
        p["ybias"] -= rated * lr("lr_yb") * sums(self.ge[:, None], self.u)
        if day:
            d = sums(self.seqd / self.nd[:, None], self.run)
            p["yfeat_day"] -= rated * lr("lr_yd") * (d + lr("reg_yd") * p["yfeat_day"])
        self.cache()
        order = torch.argsort(self.i, stable=True)
        icnt = torch.bincount(self.i, minlength=I)
        ioff = torch.cat([icnt.new_zeros(1), icnt.cumsum(0)])
        items = torch.argsort(icnt, descending=True)
        steps = icnt[items].cpu().numpy()
        for k in range(int(steps[0])):
            m = int(np.searchsorted(-steps, -k, side="left"))
            i = items[:m]
            t = order[ioff[i] + k]
            u, tb, ud, dv, fb = self.u[t], self.tb[t], self.ud[t], self.dev[t], self.fb[t]
            pe = p["ufeat"][u] + p["ycache"][u] + dv[:, None] * p["ufeat2"][u]
            if day:
                pe = pe + p["ufeat_day"][ud] + p["ycache_day"][ud]
            q, qf, cu = p["ifeat"][i], p["ifeat_freq"][i * NF + fb], p["cu"][u, 0]
            bi = p["ibias"][i, 0] + p["bit_bin"][i, tb] + p["ibias_freq"][i, fb]
            score = (self.gbias + p["ubias"][u, 0] + p["but_bin"][u, tb] + p["alpha_u"][u, 0] * dv
                     + p["ubias_day"][ud, 0] + p["ycache_bias"][u, 0] + bi * cu + (pe * (q + qf)).sum(1))
            e = self.err(score, self.res[t])
            p["ibias"][i, 0] -= lr("lr_ib") * e * cu
            p["bit_bin"][i, tb] -= lr("lr_ti") * e * cu
            p["ibias_freq"][i, fb] -= lr("lr_ibf") * e * cu
            ep = e[:, None] * pe
            p["ifeat"][i] -= lr("lr_i") * (ep + lr("reg_i") * q)
            p["ifeat_freq"][i * NF + fb] -= lr("lr_iqf") * (ep + lr("reg_iqf") * qf)

    def predict(self, u, i, day):
        p, NF, day_on = self.p, self.c.n_freq_bins, self.case["per_day"]
        tb, dv = self.tbin(day), self.dev_of(u, day)
        ud = torch.searchsorted(self.ud_key, u * 4096 + day).clamp(max=len(self.ud_key) - 1)
        has = self.ud_key[ud] == u * 4096 + day
        fb = torch.where(has, self.bin_of_ud[ud], torch.zeros_like(ud))
        pe = p["ufeat"][u] + p["ycache"][u] + dv[:, None] * p["ufeat2"][u]
        if day_on:
            pe = pe + (p["ufeat_day"][ud] + p["ycache_day"][ud]) * has[:, None]
        bi = p["ibias"][i, 0] + p["bit_bin"][i, tb] + p["ibias_freq"][i, fb]
        return (self.gbias + p["ubias"][u, 0] + p["but_bin"][u, tb] + p["alpha_u"][u, 0] * dv
                + has * p["ubias_day"][ud, 0] + p["ycache_bias"][u, 0] + bi * p["cu"][u, 0]
                + (pe * (p["ifeat"][i] + p["ifeat_freq"][i * NF + fb])).sum(1))

    def encoder(self, seed):
        """One AdamW epoch of the encoder over the case's users."""
        case, p, T = self.case, self.p, self.c.n_time_bins
        users = torch.from_numpy(_some_users(case, seed).astype(np.int64)).to(self.u.device)
        w = {n: v.double().requires_grad_() for n, v in _enc_values(case, seed).items()}
        target = torch.cat([p["ufeat"], p["ubias"], p["alpha_u"]], 1)[users]
        target = (target - target.mean(0)) / target.std(0, unbiased=False)
        mom = {n: [torch.zeros_like(v), torch.zeros_like(v)] for n, v in w.items()}
        total, steps = 0.0, 0
        gelu = torch.nn.functional.gelu
        for a in range(0, len(users), case["batch"]):
            b = users[a:a + case["batch"]]
            t = torch.cat([torch.arange(int(self.off[x]), int(self.off[x + 1]), device=b.device) for x in b.tolist()])
            at = torch.repeat_interleave(torch.arange(len(b), device=b.device), self.cnt[b])
            r = self.res[t].long() - 1
            rows = w["e_item"][self.i[t] * 5 + r] + w["e_rate"][r] + w["e_date"][self.tb[t]]
            h = torch.zeros((len(b), 128), device=b.device, dtype=torch.float64).index_add(0, at, rows)
            h = h / self.cnt[b].clamp(min=1)[:, None]
            h = gelu(h @ w["w1"] + w["b1"][:, 0])
            h = gelu(h @ w["w2"] + w["b2"][:, 0])
            loss = ((h @ w["w3"] + w["b3"][:, 0] - target[a:a + len(b)]) ** 2).mean()
            grads = torch.autograd.grad(loss, list(w.values()))
            steps += 1
            total += loss.item()
            with torch.no_grad():
                for (n, v), g in zip(w.items(), grads):
                    m1, m2 = mom[n]
                    m1.mul_(0.9).add_(0.1 * g)
                    m2.mul_(0.999).add_(0.001 * g * g)
                    up = (m1 / (1 - 0.9 ** steps)) / (torch.sqrt(m2 / (1 - 0.999 ** steps)) + 1e-8)
                    v -= 1e-4 * (up + (1e-4 * v if n in ("w1", "w2", "w3") else 0.0))
        shape = lambda n, v: v.detach()[:, 0] if n in ("b1", "b2", "b3") else v.detach()
        return {"loss": total / steps, **{n: shape(n, v).cpu().numpy() for n, v in w.items()}}


def exact(case, seed):
    """None where the item and user chains, taken a step at a time, would be too long."""
    kind = case["kind"]
    cols = _columns(case, seed)
    if kind in ("epoch", "group", "foldin"):
        t = cols[0]
        longest = int(torch.bincount(t["u"]).max()) * (case["passes"] or 1)
        if kind != "foldin":
            longest += int(torch.bincount(t["i"]).max())
        if longest * max(1, case["variants"]) > 50_000 or case["ratings"] * case["f"] > 1e9:
            return None
    if kind == "group":
        got = []
        for k in range(case["variants"]):
            x = _Exact(case, seed + k, cols, k)
            x.epoch()
            got.append(x.out())
        return got
    x = _Exact(case, seed, cols)
    if kind == "epoch":
        x.epoch()
        return x.out()
    if kind == "encoder":
        return x.encoder(seed)
    x.cache()
    if kind == "foldin":
        users = torch.from_numpy(_some_users(case, seed).astype(np.int64)).to(x.u.device)
        for _ in range(case["passes"]):
            x.users_pass(users[x.cnt[users] > 0])
        return x.out(USER_TABLES)
    u, i, day = (v.long() for v in _query(case, seed))
    step = 1 << 17
    got = torch.cat([x.predict(u[a:a + step], i[a:a + step], day[a:a + step]) for a in range(0, len(u), step)])
    if kind == "predict":
        return got
    target = (1 + (u.int() * 7 + i.int() * 13) % 5).double()
    return {"pred": got.cpu().numpy(), "rmse": float(torch.sqrt(((got - target) ** 2).mean()))}
