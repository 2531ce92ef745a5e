"""GROUP BY keys of many values (the record table with its block cache of hot
keys, groups ordered by a bitmap of their first rows) against the oracle:
group order, counts, integer sums, minima and maxima exactly, float64 sums
and averages against the exact values."""

import numpy as np
import pytest

from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.plan import (Avg, ColRef, ColRefE, Count, GroupByAggregateOperator, Lt, Literal, Max, Min,
                              OperatorSchema, OrderByOperator, OutputOperator, ScanOperator, SelectOperator, Sum, Type,
                              VirtColRef)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _keys(rng, kind, rows):
    """(type, values, nulls)"""
    if kind == "unique":
        return Type.Int(), rng.permutation(rows).astype(np.int32), None
    if kind == "hot":  # half the rows share a key, the rest are spread out
        k = rng.integers(0, max(rows // 2, 1), rows)
        k[rng.random(rows) < 0.5] = 7
        return Type.Int(), k.astype(np.int32), None
    if kind == "few":
        return Type.SmallInt(), rng.integers(-3, 3, rows).astype(np.int16), None
    if kind == "null":
        return Type.Int(), rng.integers(0, 40, rows).astype(np.int32), (rng.random(rows) < 0.3).astype(np.int8)
    # BIGINT: the value 0 (which marks an empty record) and both ends of the range among the keys
    pool = np.concatenate([np.array([0, -1, 1, 2**63 - 1, -2**63]), rng.integers(-2**62, 2**62, 200)])
    k = pool[rng.integers(0, len(pool), rows)]
    return Type.BigInt(), k, (rng.random(rows) < 0.1).astype(np.int8) if kind == "bigint_null" else None


def _table(name, kind, rows):
    rng = np.random.default_rng(rows + len(kind))
    typ, k, nulls = _keys(rng, kind, rows)
    t = HostTable(name)
    t.add(HostColumn("k", typ, values=k, nulls=nulls))
    t.add(HostColumn("v", Type.Real(), values=rng.random(rows) * 1000 - 300, nulls=(rng.random(rows) < 0.2).astype(np.int8)))
    t.add(HostColumn("d", Type.Date(), values=rng.integers(2440588, 2450000, rows).astype(np.int32)))
    t.add(HostColumn("i", Type.BigInt(), values=rng.integers(-2**40, 2**40, rows)))
    return t


def _plan(t, having=False, ordered=False, text=False):
    rel = catalog_of([t])[t.name]
    s = OperatorSchema()
    s.AddGeneratedColumns(rel, list(t.columns))
    src = ScanOperator(s, rel)
    if having:
        f = OperatorSchema()
        f.AddPassthroughColumns(src)
        src = SelectOperator(f, src, Lt(ColRef(src, "d"), ColRef(src, "d")))
    key = ColRefE(src, "k")
    aggs = [Sum(ColRef(src, "v")), Min(ColRef(src, "d")), Count(), Max(ColRef(src, "v")), Sum(ColRef(src, "i")),
            Count(ColRef(src, "v")), Avg(ColRef(src, "v"))]
    if text:
        aggs = aggs[:3] + [Min(ColRef(src, "s")), Max(ColRef(src, "s"))]
    o = OperatorSchema()
    o.AddDerivedColumn("k", VirtColRef(key, 0))
    for i, a in enumerate(aggs):
        o.AddDerivedColumn(f"a{i}", VirtColRef(a, i + 1))
    g = GroupByAggregateOperator(o, src, [key], aggs)
    if not ordered:
        return OutputOperator(g)
    oo = OperatorSchema()
    oo.AddPassthroughColumns(g)
    return OutputOperator(OrderByOperator(oo, g, [ColRef(g, "a2")], [False]))


def _check(engine, t, plan):
    """Everything but the sums and averages of `v` equals the oracle's; those
    are within the rounding of n additions in any order, n * eps * sum|v|, of
    the exact value (the oracle's running average is itself further off where
    values of both signs cancel)."""
    from oracle import Oracle
    o = Oracle()
    o.register_table(t)
    engine.register_table(t)
    ref = o.execute(plan)
    v = t.columns["v"]
    k = t.columns["k"]
    kn = np.zeros(len(k), np.int8) if k.nulls is None else k.nulls
    member = np.where(kn != 0, -1, np.unique(k.values, return_inverse=True)[1])
    first = {}
    for _ in range(3):  # fresh, recorded, replayed
        g = engine.execute(plan)
        assert len(g.columns) == len(ref.columns) and g.num_rows == ref.num_rows
        for c, (x, y) in enumerate(zip(g.columns, ref.columns)):
            assert np.array_equal(x.nulls, y.nulls), f"column {c}: nulls"
            live = np.asarray(y.nulls) == 0
            if c not in (1, 7):  # SUM(v), AVG(v)
                assert np.array_equal(np.asarray(x.values)[live], np.asarray(y.values)[live]), f"column {c}"
        if not first and g.num_rows:
            ids = {}
            for i, (kv, nul) in enumerate(zip(k.values.tolist(), kn.tolist())):
                ids.setdefault(None if nul else kv, member[i])
            at = np.array([ids[None if n else int(kv)] for kv, n in zip(g.columns[0].values, g.columns[0].nulls)])
            n_ids = int(member.max()) + 2
            vals = np.where(v.nulls != 0, 0.0, v.values).astype(np.longdouble)
            total, size, count = np.zeros(n_ids, np.longdouble), np.zeros(n_ids, np.longdouble), np.zeros(n_ids)
            np.add.at(total, member, vals)
            np.add.at(size, member, np.abs(vals))
            np.add.at(count, member, v.nulls == 0)
            first = {"at": at, "total": total, "size": size, "count": count}
        if first:
            at = first["at"]
            n = np.maximum(first["count"][at], 1)
            bound = n * 2.0 ** -52 * first["size"][at]
            live = np.asarray(g.columns[1].nulls) == 0
            assert np.all(np.abs(g.columns[1].values - first["total"][at])[live] <= bound[live]), "SUM(v)"
            if len(g.columns) > 7:
                assert np.all(np.abs(g.columns[7].values - first["total"][at] / n)[live] <= (bound / n)[live] * 2), "AVG(v)"


# around a bitmap word (32 rows), a chunk of the order (32768 rows), the
# block cache (1024 keys) and one CTA's rows
@pytest.mark.parametrize("rows", [1, 31, 33, 1023, 1025, 32_768, 32_769, 150_001])
@pytest.mark.parametrize("kind", ["unique", "hot", "few", "null", "bigint", "bigint_null"])
def test_group_keys_match_oracle(engine, rows, kind):
    t = _table(f"gk_{kind}_{rows}", kind, rows)
    _check(engine, t, _plan(t))


@pytest.mark.parametrize("kind", ["hot", "bigint"])
def test_group_keys_under_order_by_match_oracle(engine, kind):
    # COUNT ties: equal keys come in the reference's merge order of the groups' first appearance
    t = _table(f"gko_{kind}", kind, 60_001)
    _check(engine, t, _plan(t, ordered=True))


def test_group_keys_empty_input(engine):
    t = _table("gk_none", "hot", 5000)
    _check(engine, t, _plan(t, having=True))


def test_group_keys_text_extremes(engine):
    t = _table("gk_text", "hot", 20_011)
    rng = np.random.default_rng(4)
    t.add(HostColumn.from_strings("s", ["".join(chr(97 + c) for c in rng.integers(0, 5, rng.integers(0, 9)))
                                        for _ in range(20_011)]))
    _check(engine, t, _plan(t, text=True))
