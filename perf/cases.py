"""Performance cases: the queries and operators that a user of the engine runs.

Every case goes through the public Python API (``Engine.execute``,
``Batch``, ``HashTable``, ``JoinPriorModel``) over tables that stay resident
in one engine, the way a program that serves queries holds them.  Sizes and
value distributions are those of ``kushdb_b200/workloads.py`` and
``bench.py`` (TPC-H Q6 / Q1 / Q3 shapes, the per-operator hash join, the
batched template, JOB-style multiway joins, the join-order prior), scaled
from the small tables of the end-to-end tests up to tables far larger than
the L2 cache.  Inputs are generated on the GPU from the seed; filters pass a
fixed number of rows and every key occurs, so that results of one case have
one size whatever the seed.

Kinds:

* ``scan_agg``    filter + ungrouped aggregate (Q6 shape): the smallest query
  a program sends, where launches and latency count, up to a scan that is
  bound by memory bandwidth;
* ``group_by``    filter + GROUP BY two ENUM keys + ORDER BY (Q1 shape);
* ``group_keys``  GROUP BY an INT or BIGINT column of many distinct values,
  uniform or skewed, result in first-appearance order;
* ``join_group``  hash join + GROUP BY the build key + ORDER BY (Q3 shape),
  uniform or skewed foreign keys;
* ``order_by``    filter + ORDER BY a REAL or DATE column, all rows returned;
* ``hash_join``   the hash join operator by itself: build, probe, pairs;
* ``batched``     many small queries of one template in one CUDA graph, with
  every query's result read back;
* ``skinner``     a 6 to 8 table join with LIKE filters through the Skinner
  join (star or chain, uniform or skewed foreign keys);
* ``prior``       forward and backward of the learned join-order prior.
"""

import math

import numpy as np
import torch

from kushdb_b200 import workloads as wl
from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.engine import Batch, Engine, JoinPriorModel
from kushdb_b200.operators import HashTable
from kushdb_b200.plan import (EPOCH_JDN, ColRef, ColRefE, Count, GroupByAggregateOperator, LiteralExpression, Lt, Min,
                              OperatorSchema, OrderByOperator, OutputOperator, ScanOperator, ScanSelectOperator, Sum,
                              Type, VirtColRef)

DATE_LO, DATE_HI = 8035, 10591          # the generators' date range (days since 1970-01-01)
SKINNER_BUDGET = 100_000                # tuples examined per episode, as in bench.py


def listed():
    return [
        # a dashboard tile over a small table: latency and launches
        {"name": "scan_agg_60k", "kind": "scan_agg", "rows": 60_175},
        # a full scan of a table ten times the L2 cache
        {"name": "scan_agg_64m", "kind": "scan_agg", "rows": 64_000_003},
        # TPC-H Q1 at SF1: few groups, many aggregates
        {"name": "group_by_6m", "kind": "group_by", "rows": 6_000_000},
        # per-customer totals: many groups, skewed customers
        {"name": "group_keys_3m", "kind": "group_keys", "rows": 3_000_017, "keys": 200_003, "type": "INT",
         "zipf": True},
        # TPC-H Q3 at SF1
        {"name": "join_group_6m", "kind": "join_group", "build": 1_500_000, "probe": 6_000_000, "zipf": False},
        # the same query over a small, skewed data set
        {"name": "join_group_zipf_400k", "kind": "join_group", "build": 100_003, "probe": 400_009, "zipf": True},
        # a sorted report: about half the rows come back
        {"name": "order_by_2m", "kind": "order_by", "rows": 2_000_003, "key": "REAL"},
        # a host program driving one join by itself
        {"name": "hash_join_6m", "kind": "hash_join", "build": 6_000_013, "probe": 3_000_017},
        # many uneven tenant queries of one template
        {"name": "batched_24", "kind": "batched", "queries": 24, "max_fact": 2_000_000},
        # JOB-style star join, uniform keys, large tables
        {"name": "skinner_star6", "kind": "skinner", "shape": "star", "tables": 6, "max_rows": 3_000_000,
         "zipf": False},
        # JOB-style chain join, skewed keys, medium tables
        {"name": "skinner_chain7_zipf", "kind": "skinner", "shape": "chain", "tables": 7, "max_rows": 300_000,
         "zipf": True},
        # one training batch of the join-order prior
        {"name": "prior_512", "kind": "prior", "rows": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan_agg", "group_by", "group_keys", "join_group", "order_by", "hash_join", "batched",
                       "skinner", "prior"])
    if kind == "scan_agg":
        return {"kind": kind, "rows": _log_int(rng, 10_000, 64_000_000)}
    if kind == "group_by":
        return {"kind": kind, "rows": _log_int(rng, 10_000, 6_000_000)}
    if kind == "group_keys":
        rows = _log_int(rng, 10_000, 3_000_000)
        return {"kind": kind, "rows": rows, "keys": _log_int(rng, 100, max(101, min(rows // 4, 200_000))),
                "type": rng.choice(["INT", "BIGINT"]), "zipf": rng.random() < 0.5}
    if kind == "join_group":
        build = _log_int(rng, 5_000, 1_500_000)
        return {"kind": kind, "build": build, "probe": _log_int(rng, 2 * build, 4 * build), "zipf": rng.random() < 0.5}
    if kind == "order_by":
        return {"kind": kind, "rows": _log_int(rng, 10_000, 2_000_000), "key": rng.choice(["REAL", "DATE"])}
    if kind == "hash_join":
        return {"kind": kind, "build": _log_int(rng, 10_000, 6_000_000), "probe": _log_int(rng, 10_000, 3_000_000)}
    if kind == "batched":
        return {"kind": kind, "queries": rng.randint(4, 24), "max_fact": _log_int(rng, 50_000, 2_000_000)}
    if kind == "skinner":
        zipf = rng.random() < 0.5
        return {"kind": kind, "shape": rng.choice(["star", "chain"]), "tables": rng.randint(6, 8),
                "max_rows": _log_int(rng, 30_000, 300_000 if zipf else 1_000_000), "zipf": zipf}
    return {"kind": kind, "rows": _log_int(rng, 16, 4096)}


# ---------------------------------------------------------------------------
# inputs (seeded, generated on the GPU)
# ---------------------------------------------------------------------------


class _Gen:
    """Column generators with the distributions of kushdb_b200/workloads.py."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def uniform(self, n):
        return torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64)

    def ints(self, n, lo, hi_inclusive, dtype=torch.int32):
        return torch.randint(lo, hi_inclusive + 1, (n,), generator=self.g, device="cuda", dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")

    def price(self, n):
        return 900.0 + self.uniform(n) * 104100.0

    def hundredths(self, n, hi):
        return self.ints(n, 0, hi).double() / 100.0

    def dates(self, n):
        return self.ints(n, DATE_LO + EPOCH_JDN, DATE_HI + EPOCH_JDN)

    def spread_dates(self, n):
        """The date range spread evenly over n rows, in random order: a date bound passes a fixed number of rows."""
        return (DATE_LO + EPOCH_JDN + self.perm(n) * (DATE_HI - DATE_LO + 1) // n).int()

    def all_keys(self, n, nkeys, zipf):
        """keys() in which each of the nkeys occurs (n >= nkeys), in random order."""
        k = torch.cat([torch.arange(nkeys, device="cuda"), self.keys(n - nkeys, nkeys, zipf)])
        return k[self.perm(n)]

    def keys(self, n, nkeys, zipf, s=1.0):
        """Indices in [0, nkeys): uniform, or Zipf(s) over permuted ranks."""
        if not zipf:
            return self.ints(n, 0, nkeys - 1, torch.int64)
        w = torch.arange(1, nkeys + 1, device="cuda", dtype=torch.float64).pow(-s)
        cdf = torch.cumsum(w, 0)
        ranks = torch.searchsorted(cdf / cdf[-1], self.uniform(n), right=True).clamp_(max=nkeys - 1)
        return self.perm(nkeys)[ranks]


def _scan_agg_inputs(case, seed):
    n, g = case["rows"], _Gen(seed)
    return {"s_price": g.price(n), "s_discount": g.hundredths(n, 10), "s_date": g.dates(n)}


def _group_by_inputs(case, seed):
    n, g = case["rows"], _Gen(seed)
    grp = g.ints(n, 0, len(wl.GROUPS) - 1, torch.int64)
    rf = torch.tensor([wl.RF_VALUES.index(a) for a, _ in wl.GROUPS], dtype=torch.int32, device="cuda")
    ls = torch.tensor([wl.LS_VALUES.index(b) for _, b in wl.GROUPS], dtype=torch.int32, device="cuda")
    return {"l_shipdate": g.dates(n), "l_returnflag": rf[grp], "l_linestatus": ls[grp],
            "l_quantity": g.ints(n, 1, 50).double(), "l_extendedprice": g.price(n),
            "l_discount": g.hundredths(n, 10), "l_tax": g.hundredths(n, 8)}


def _group_keys_inputs(case, seed):
    n, g = case["rows"], _Gen(seed)
    k = g.all_keys(n, case["keys"], case["zipf"])
    # BIGINT keys are sparse, as surrogate keys of a partitioned source are
    k = k * 1_000_003 + 77 if case["type"] == "BIGINT" else (k + 1).int()
    return {"s_key": k, "s_price": g.price(n), "s_date": g.dates(n)}


def _join_group_inputs(case, seed):
    nb, np_, g = case["build"], case["probe"], _Gen(seed)
    cell = g.perm(nb)  # segments in turn, dates spread evenly within each
    n_seg = len(wl.SEG_VALUES)
    date = DATE_LO + EPOCH_JDN + (cell // n_seg) * (DATE_HI - DATE_LO + 1) // (nb // n_seg + 1)
    build = {"c_custkey": torch.arange(1, nb + 1, dtype=torch.int32, device="cuda"), "c_date": date.int(),
             "c_segment": (cell % n_seg).int()}
    probe = {"o_custkey": (g.all_keys(np_, nb, case["zipf"]) + 1).int(), "o_price": g.price(np_),
             "o_discount": g.hundredths(np_, 10)}
    return build, probe


def _order_by_inputs(case, seed):
    n, g = case["rows"], _Gen(seed)
    return {"s_key": g.ints(n, 0, 999_999), "s_price": g.price(n), "s_date": g.dates(n),
            "s_pick": g.spread_dates(n)}


def _hash_join_inputs(case, seed):
    nb, np_, g = case["build"], case["probe"], _Gen(seed)
    # a primary key in load order, foreign keys of which a fifth have no match
    miss = g.perm(np_) < np_ // 5
    return (g.perm(nb) + 1).int(), g.ints(np_, 1, nb) + miss.int() * nb


def _batched_inputs(case, seed):
    """[(dim columns, fact columns, date bound)]: fact rows log-uniform, dimension a quarter of them."""
    g = _Gen(seed)
    out = []
    for q in range(case["queries"]):
        # sizes depend on the query's number alone, so every seed costs the same
        f = (q * 0.6180339887498949 + 0.5) % 1.0
        nf = int(10_000 * (case["max_fact"] / 10_000) ** f)
        nd = max(1, nf // 4)
        dim = {"d_key": torch.arange(nd, dtype=torch.int32, device="cuda") * 7 + q, "d_date": g.spread_dates(nd),
               "d_seg": torch.zeros(nd, dtype=torch.int32, device="cuda")}
        fact = {"f_fk": g.all_keys(nf, nd, False).int() * 7 + q, "f_price": g.price(nf), "f_disc": g.hundredths(nf, 10)}
        share = 0.01 + 0.89 * ((q * 0.7548776662466927 + 0.25) % 1.0)
        out.append((dim, fact, EPOCH_JDN + DATE_LO + int(round(share * (DATE_HI - DATE_LO + 1)))))
    return out


def _skinner_sizes(case):
    n, hi = case["tables"], case["max_rows"]
    sizes = [int(10_000 * (hi / 10_000) ** ((i * 0.6180339887498949 + 1.0) % 1.0)) for i in range(n)]
    sizes[0] = hi
    return sorted(sizes, reverse=True) if case["shape"] == "star" else sizes


def _notes(g, n, token, share):
    """n random printable strings of 8 to 40 bytes, `share` of them holding `token`."""
    lens = g.ints(n, 8, 40, torch.int64)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    alphabet = torch.from_numpy(wl.PRINTABLE.copy()).cuda()
    chars = alphabet[g.ints(int(off[-1]), 0, len(wl.PRINTABLE) - 1, torch.int64)]
    at = off[:-1] + (g.uniform(n) * (lens - len(token) + 1).double()).long()
    at = at[g.uniform(n) < share]
    for i, c in enumerate(token.encode()):
        chars[at + i] = c
    return off, chars


# ---------------------------------------------------------------------------
# preparation: resident tables and serialised plans
# ---------------------------------------------------------------------------

_engine_ = None
_serial = 0


def _engine():
    global _engine_
    if _engine_ is None:
        _engine_ = Engine(0)
        _engine_.set_skinner(SKINNER_BUDGET, 0)
        wl.register_enums()
    return _engine_


_TYPES = {torch.int32: Type.Int, torch.int64: Type.BigInt, torch.float64: Type.Real}
_ENUMS = {"l_returnflag": wl.RF_ENUM_ID, "l_linestatus": wl.LS_ENUM_ID, "c_segment": wl.SEG_ENUM_ID}
_DATES = {"s_date", "s_pick", "l_shipdate", "c_date", "d_date"}


class _State:
    """Tables registered under names of their own, and what runs over them."""

    def __init__(self, kind):
        self.kind, self.engine = kind, _engine()
        self.names, self.batch = [], None

    def table(self, name, columns, texts=()):
        global _serial
        _serial += 1
        t = HostTable("%s_%d" % (name, _serial))
        for c, v in columns.items():
            typ = Type.Enum(_ENUMS[c]) if c in _ENUMS else Type.Date() if c in _DATES else _TYPES[v.dtype]()
            t.add(HostColumn(c, typ, values=v.cpu().numpy()))
        for c, (off, chars) in dict(texts).items():
            t.add(HostColumn(c, Type.Text(), offsets=off.cpu().numpy(), chars=chars.cpu().numpy()))
        self.engine.register_table(t)
        self.names.append(t.name)
        return t

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for n in self.names:
            self.engine.drop_table(n)


def _text(plan):
    return plan.to_json().encode()


def _group_keys_plan(t):
    rel = catalog_of([t])[t.name]
    scan = OperatorSchema()
    scan.AddGeneratedColumns(rel, ["s_key", "s_price", "s_date"])
    src = ScanOperator(scan, rel)
    key = ColRefE(src, "s_key")
    aggs = [Sum(ColRef(src, "s_price")), Min(ColRef(src, "s_date")), Count()]
    out = OperatorSchema()
    out.AddDerivedColumn("s_key", VirtColRef(key, 0))
    for i, n in enumerate(["total", "first_date", "orders"]):
        out.AddDerivedColumn(n, VirtColRef(aggs[i], i + 1))
    return OutputOperator(GroupByAggregateOperator(out, src, [key], aggs))


ORDER_BY_DATE_LT = (DATE_LO + DATE_HI) // 2


def _order_by_plan(t, key):
    rel = catalog_of([t])[t.name]
    scan = OperatorSchema()
    scan.AddGeneratedColumns(rel, ["s_key", "s_price", "s_date", "s_pick"])
    keep = Lt(VirtColRef(scan, "s_pick"), LiteralExpression(Type.Date(), ORDER_BY_DATE_LT + EPOCH_JDN))
    out = OperatorSchema()
    out.AddVirtualPassthroughColumns(scan, ["s_key", "s_price", "s_date"])
    sel = ScanSelectOperator(out, scan, rel, [keep])
    o = OperatorSchema()
    o.AddPassthroughColumns(sel)
    by = "s_price" if key == "REAL" else "s_date"
    return OutputOperator(OrderByOperator(o, sel, [ColRef(sel, by)], [True]))


def prepare(case, seed):
    kind = case["kind"]
    s = _State(kind)
    if kind == "scan_agg":
        s.plan = _text(wl.scan_agg_plan(s.table("sales", _scan_agg_inputs(case, seed))))
    elif kind == "group_by":
        s.plan = _text(wl.group_by_plan(s.table("lineitem", _group_by_inputs(case, seed))))
    elif kind == "group_keys":
        s.plan = _text(_group_keys_plan(s.table("sales", _group_keys_inputs(case, seed))))
    elif kind == "join_group":
        build, probe = _join_group_inputs(case, seed)
        s.plan = _text(wl.join_plan(s.table("customer", build), s.table("orders", probe)))
    elif kind == "order_by":
        s.plan = _text(_order_by_plan(s.table("sales", _order_by_inputs(case, seed)), case["key"]))
    elif kind == "hash_join":
        build, probe = _hash_join_inputs(case, seed)
        s.build = s.table("build", {"k": build}).name
        s.probe = s.table("probe", {"k": probe}).name
    elif kind == "batched":
        descs = []
        for dim, fact, date_lt in _batched_inputs(case, seed):
            d, f = s.table("dim", dim), s.table("fact", fact)
            descs.append(wl.batch_query_desc(d, f, date_lt, 0))
        s.batch = Batch(s.engine, descs)
    elif kind == "skinner":
        s.plan = _text(_skinner(s, case, seed))
    else:
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        s.model = JoinPriorModel(s.engine, seed=seed & 0xffff)
        # features are shares and logarithms of cardinalities, rewards in [0, 1]
        s.x = torch.rand(case["rows"], s.model.num_features, generator=g, device="cuda").cpu().numpy()
        s.t = torch.rand(case["rows"], generator=g, device="cuda").cpu().numpy()
    s.engine.register_enums()
    return s


def _skinner(s, case, seed):
    g, sizes = _Gen(seed), _skinner_sizes(case)
    tables, tokens = [], []
    for i, n in enumerate(sizes):
        token = "".join(chr(97 + int(c)) for c in g.ints(3, 0, 25).tolist())
        tokens.append(token)
        cols = {"pk": torch.arange(n, dtype=torch.int32, device="cuda")}
        if case["shape"] == "star":
            if i == 0:
                for j in range(1, len(sizes)):
                    cols["fk%d" % j] = g.keys(n, sizes[j], case["zipf"], 1.5).int()
        elif i > 0:
            cols["fk"] = g.keys(n, sizes[i - 1], case["zipf"], 1.5).int()
        tables.append(s.table("t%d" % i, cols, {"note": _notes(g, n, token, 0.06)}))
    # the filters sit on two dimensions of a star, on the two last links of a chain
    like = (1, 2) if case["shape"] == "star" else (len(sizes) - 2, len(sizes) - 1)
    return wl.skinner_plan(tables, tokens, case["shape"], like)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(state):
    e = state.engine
    if state.kind == "hash_join":
        ht = HashTable(e, state.build, "k")
        rows = ht.probe(state.probe, "k")
        ht.close()
        return {"probe_rows": rows[0], "build_rows": rows[1]}
    if state.kind == "batched":
        state.batch.run()
        res = [state.batch.result(q) for q in range(state.batch.n)]
        return {"keys": np.concatenate([k for k, _ in res]), "sums": np.concatenate([v for _, v in res]),
                "groups": np.array([len(k) for k, _ in res])}
    if state.kind == "prior":
        grad, loss = state.model.gradient(state.x, state.t)
        return {"gradient": grad, "loss": loss}
    return [c.values for c in e.execute(state.plan).columns]


# ---------------------------------------------------------------------------
# 64-bit values of the outputs, in plain torch
# ---------------------------------------------------------------------------


def _sums(values, group, ngroups):
    return torch.zeros(ngroups, dtype=torch.float64, device="cuda").index_add_(0, group, values)


def exact(case, seed):
    kind = case["kind"]
    if kind == "scan_agg":
        c = _scan_agg_inputs(case, seed)
        m = (c["s_date"] < 9300 + EPOCH_JDN) & (c["s_discount"] >= 0.05) & (c["s_discount"] <= 0.07)
        return [(c["s_price"][m] * c["s_discount"][m]).sum().reshape(1), None]
    if kind == "group_by":
        c = _group_by_inputs(case, seed)
        m = c["l_shipdate"] <= 10471 + EPOCH_JDN
        c = {k: v[m] for k, v in c.items()}
        # both dictionaries are in string order, so the codes order the output
        _, grp = torch.unique(c["l_returnflag"].long() * 16 + c["l_linestatus"].long(), return_inverse=True)
        n = int(grp.max()) + 1
        cnt = torch.bincount(grp, minlength=n).double()
        net = c["l_extendedprice"] * (1.0 - c["l_discount"])
        qty, base = _sums(c["l_quantity"], grp, n), _sums(c["l_extendedprice"], grp, n)
        return [None, None, qty, base, _sums(net, grp, n), _sums(net * (1.0 + c["l_tax"]), grp, n), qty / cnt,
                base / cnt, _sums(c["l_discount"], grp, n) / cnt, None]
    if kind == "group_keys":
        c = _group_keys_inputs(case, seed)
        _, grp = torch.unique(c["s_key"], return_inverse=True)
        n = int(grp.max()) + 1
        first = torch.full((n,), case["rows"], dtype=torch.int64, device="cuda")
        first.scatter_reduce_(0, grp, torch.arange(case["rows"], device="cuda"), "amin")
        return [None, _sums(c["s_price"], grp, n)[torch.argsort(first)], None, None]
    if kind == "join_group":
        b, p = _join_group_inputs(case, seed)
        keep = (b["c_date"] < 9204 + EPOCH_JDN) & (b["c_segment"] == wl.SEG_VALUES.index("BUILDING"))
        fk = p["o_custkey"].long() - 1
        m = keep[fk]
        rev = _sums((p["o_price"] * (1.0 - p["o_discount"]))[m], fk[m], case["build"])
        hit = torch.bincount(fk[m], minlength=case["build"]) > 0
        return [None, torch.sort(rev[hit], descending=True).values]
    if kind == "order_by" and case["key"] == "REAL":
        c = _order_by_inputs(case, seed)
        return [None, torch.sort(c["s_price"][c["s_pick"] < ORDER_BY_DATE_LT + EPOCH_JDN]).values, None]
    if kind == "batched":
        sums = []
        for dim, fact, date_lt in _batched_inputs(case, seed):
            ref = ((fact["f_fk"] - dim["d_key"][0]) // 7).long()
            m = (dim["d_date"] < date_lt)[ref]
            ref, rev = ref[m], (fact["f_price"] * (1.0 - fact["f_disc"]))[m]
            uniq, grp = torch.unique(ref, return_inverse=True)
            first = torch.full((len(uniq),), len(ref), dtype=torch.int64, device="cuda")
            first.scatter_reduce_(0, grp, torch.arange(len(ref), device="cuda"), "amin")
            sums.append(_sums(rev, grp, len(uniq))[torch.argsort(first)])
        return {"keys": None, "sums": torch.cat(sums), "groups": None}
    if kind == "prior":
        s = prepare(case, seed)
        p = torch.from_numpy(s.model.params()).double().cuda().requires_grad_(True)
        h, at = torch.from_numpy(s.x).double().cuda(), 0
        for fan_in, fan_out in ((64, 128), (128, 128), (128, 128), (128, 1)):
            w = p[at:at + fan_in * fan_out].reshape(fan_in, fan_out)
            at += fan_in * fan_out
            h = h @ w + p[at:at + fan_out]
            at += fan_out
            if fan_out > 1:
                h = torch.relu(h)
        loss = (h[:, 0] - torch.from_numpy(s.t).double().cuda()).square().mean()
        loss.backward()
        return {"gradient": p.grad.detach(), "loss": float(loss)}
    return None  # only whole numbers come back, or their order alone decides the values


# ---------------------------------------------------------------------------
# work one pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "scan_agg":
        return {"bytes": case["rows"] * 20, "flops": case["rows"] * 2}
    if kind == "group_by":
        return {"bytes": case["rows"] * 44, "flops": case["rows"] * 12}
    if kind == "group_keys":
        key = 8 if case["type"] == "BIGINT" else 4
        return {"bytes": case["rows"] * (key + 12) + case["keys"] * (key + 20), "flops": case["rows"]}
    if kind == "join_group":
        share = (9204 - DATE_LO) / (DATE_HI - DATE_LO + 1) / len(wl.SEG_VALUES)
        return {"bytes": case["build"] * 12 + case["probe"] * 20 + int(case["build"] * share) * 12,
                "flops": case["probe"] * 3 * share}
    if kind == "order_by":
        return {"bytes": case["rows"] * 20 + case["rows"] // 2 * 16, "flops": 0}
    if kind == "hash_join":
        return {"bytes": (case["build"] + case["probe"]) * 4 + int(case["probe"] * 0.8) * 8, "flops": 0}
    if kind == "batched":
        facts = sum(int(10_000 * (case["max_fact"] / 10_000) ** ((q * 0.6180339887498949 + 0.5) % 1.0))
                    for q in range(case["queries"]))
        return {"bytes": facts * 20 + facts // 4 * 18, "flops": facts}
    if kind == "skinner":
        # every key column once, the text of the two filtered tables once
        sizes = _skinner_sizes(case)
        keys = sum(sizes) + (sizes[0] * (len(sizes) - 1) if case["shape"] == "star" else sum(sizes[1:]))
        filtered = sizes[1] + sizes[2] if case["shape"] == "star" else sizes[-2] + sizes[-1]
        return {"bytes": 4 * keys + 32 * filtered, "flops": 0}
    weights = 64 * 128 + 2 * 128 * 128 + 128
    return {"bytes": case["rows"] * 65 * 4 + 2 * 4 * weights, "flops": 6 * case["rows"] * weights}
