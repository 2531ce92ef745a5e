"""GROUP BY where one key holds many of the rows: the values, and that such a
key costs no more than its rows would as other keys (its updates otherwise
queue on one record, one row after the other)."""

import numpy as np
import pytest

from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.plan import (AggregateOperator, ColRef, ColRefE, Count, GroupByAggregateOperator, HashJoinOperator, Max,
                              Min, OperatorSchema, OutputOperator, ScanOperator, Sum, Type, VirtColRef)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _plan(t):
    s = OperatorSchema()
    s.AddGeneratedColumns(catalog_of([t])[t.name], ["k", "v"])
    src = ScanOperator(s, catalog_of([t])[t.name])
    key = ColRefE(src, "k")
    aggs = [Sum(ColRef(src, "v")), Min(ColRef(src, "v")), Count()]
    o = OperatorSchema()
    o.AddDerivedColumn("k", VirtColRef(key, 0))
    for i, a in enumerate(aggs):
        o.AddDerivedColumn(f"a{i}", VirtColRef(a, i + 1))
    return OutputOperator(GroupByAggregateOperator(o, src, [key], aggs))


def _run(engine, name, typ, keys):
    """Checks the groups of `keys`; returns the GROUP BY kernel's time in us."""
    v = (np.arange(len(keys)) * 37 % 1009 - 500).astype(np.int32)
    t = HostTable(name)
    t.add(HostColumn("k", typ, values=keys))
    t.add(HostColumn("v", Type.Int(), values=v))
    engine.register_table(t)
    plan = _plan(t)
    got = [np.asarray(c.values) for c in engine.execute(plan).columns]
    uniq, first, member = np.unique(keys, return_index=True, return_inverse=True)
    order = np.argsort(first)
    low = np.full(len(uniq), 1 << 30, np.int64)
    np.minimum.at(low, member, v)
    want = [uniq, np.bincount(member, weights=v).astype(np.int64), low, np.bincount(member)]
    for g, w in zip(got, want):
        assert np.array_equal(g, w[order])
    engine.set_profiling(True)
    us = []
    for _ in range(5):
        engine.execute(plan, fetch=False)
        us.append(sum(k["ms"] for k in engine.last_kernels() if k["tag"] == "group by") * 1e3)
    engine.set_profiling(False)
    engine.drop_table(name)
    return sorted(us)[2]


# a row of a hot key costs at most what a row of any other key costs, and a
# factor of two for the spread of the timings
def test_hot_key_among_many_rows_per_thread(engine):
    rows = 20_000_000  # over 64 rows for each thread of the GPU
    rng = np.random.default_rng(1)
    k = rng.integers(10, 50_000, rows).astype(np.int32)
    spread = _run(engine, "hk_spread", Type.Int(), k)
    k[rng.random(rows) < 0.1] = 7
    assert _run(engine, "hk_hot", Type.Int(), k) < 2 * spread


def test_bigint_zero_is_as_cheap_as_another_hot_key(engine):
    rows = 3_000_017
    rng = np.random.default_rng(2)
    k = rng.integers(10, 200_000, rows)
    hot = rng.random(rows) < 0.5
    k[hot] = 7
    other = _run(engine, "hk_seven", Type.BigInt(), k)
    k[hot] = 0
    assert _run(engine, "hk_zero", Type.BigInt(), k) < 2 * other


def test_records_beyond_l2(engine):
    # 2M groups: the table regrows past L2, where only first positions are read ahead
    k = np.random.default_rng(3).permutation(np.concatenate([np.arange(2_000_000), np.arange(2_000_000)]))
    _run(engine, "hk_many", Type.Int(), k.astype(np.int32))
    _run(engine, "hk_many_big", Type.BigInt(), k * 5)


def _join_tables(prefix, nb, np_, dup, text):
    rng = np.random.default_rng(nb + dup)
    b, p = HostTable(prefix + "b"), HostTable(prefix + "p")
    bk, pk = rng.permutation(nb) // dup, rng.integers(-nb // (8 * dup), nb // dup, np_)
    for t, name, k in ((b, "bk", bk), (p, "pk", pk)):
        if text:
            t.add(HostColumn.from_strings(name, ["k%d" % x for x in k]))
        else:
            t.add(HostColumn(name, Type.Int(), values=k.astype(np.int32), nulls=(rng.random(len(k)) < 0.05).astype(np.int8)))
    b.add(HostColumn("bg", Type.Int(), values=rng.integers(0, 900, nb).astype(np.int32)))
    p.add(HostColumn("g", Type.Int(), values=rng.integers(0, 300, np_).astype(np.int32)))
    p.add(HostColumn("big", Type.BigInt(), values=rng.integers(0, 3, np_)))
    p.add(HostColumn("v", Type.Int(), values=rng.integers(-1000, 1000, np_).astype(np.int32)))
    return b, p


def _over_join(b, p, key):
    db = catalog_of([b, p])
    scans = []
    for t in (b, p):
        s = OperatorSchema()
        s.AddGeneratedColumns(db[t.name], list(t.columns))
        scans.append(ScanOperator(s, db[t.name]))
    js = OperatorSchema()
    js.AddPassthroughColumns(scans[0], ["bg"], 0)
    js.AddPassthroughColumns(scans[1], ["g", "big", "v"], 1)
    j = HashJoinOperator(js, scans[0], scans[1], [ColRef(scans[0], "bk", 0)], [ColRef(scans[1], "pk", 1)])
    return _groups(j, key)


def _groups(src, key):
    aggs = [Sum(ColRef(src, "v")), Min(ColRef(src, "v")), Max(ColRef(src, "v")), Count()]
    o = OperatorSchema()
    k = ColRefE(src, key) if key else None
    if key:
        o.AddDerivedColumn("k", VirtColRef(k, 0))
    for i, a in enumerate(aggs):
        o.AddDerivedColumn(f"a{i}", VirtColRef(a, i + (1 if key else 0)))
    return OutputOperator(GroupByAggregateOperator(o, src, [k], aggs) if key else AggregateOperator(o, src, aggs))


# several build rows per key, slots that share a hash (TEXT keys are compared after it), rows without a match
@pytest.mark.parametrize("dup", [1, 3])
@pytest.mark.parametrize("text", [False, True])
@pytest.mark.parametrize("key", ["bg", "g", "big"])
def test_groups_over_a_join_match_oracle(engine, dup, text, key):
    from oracle import Oracle
    from parity import compare
    b, p = _join_tables(f"gj{dup}{text}{key}", 6000, 50_011, dup, text)
    o = Oracle()
    for t in (b, p):
        engine.register_table(t)
        o.register_table(t)
    plan = _over_join(b, p, key)
    assert compare(engine.execute(plan), o.execute(plan)) == ""


# the groups of a join's matches cost about the join and the groups of as many
# rows of a table (half as much again for the spread of the timings)
def test_groups_over_a_join_cost_the_join_and_the_groups(engine):
    b, p = _join_tables("gt", 200_000, 2_000_000, 1, False)
    for t in (b, p):
        engine.register_table(t)
    s = OperatorSchema()
    s.AddGeneratedColumns(catalog_of([p])[p.name], ["g", "v"])
    plans = [_over_join(b, p, "g"), _over_join(b, p, None), _groups(ScanOperator(s, catalog_of([p])[p.name]), "g")]
    us = []
    for plan in plans:
        engine.execute(plan)
        engine.set_profiling(True)
        t = []
        for _ in range(5):
            engine.execute(plan, fetch=False)
            t.append(sum(k["ms"] for k in engine.last_kernels() if k["tag"] in ("group by", "aggregate")) * 1e3)
        engine.set_profiling(False)
        us.append(sorted(t)[2])
    assert us[0] < 1.5 * (us[1] + us[2])


# MIN / MAX of a string keeps the block cache out: a hot key's other states are
# folded all the same.  (Its strings still meet in one word: a row costs up to
# ten times what a row of any other key does; unfolded it was 45 times.)
def test_hot_key_with_string_extremes(engine):
    from oracle import Oracle
    from parity import compare
    rows = 1_000_003
    rng = np.random.default_rng(4)
    strings = ["m%04d" % x for x in rng.integers(0, 9999, rows)]
    us = []
    for name, share in (("st", 0.0), ("sh", 0.95)):
        k = rng.integers(10, 50_000, rows).astype(np.int32)
        k[rng.random(rows) < share] = 7
        t = HostTable(name)
        t.add(HostColumn("k", Type.Int(), values=k))
        t.add(HostColumn.from_strings("s", strings, (rng.random(rows) < 0.1).astype(np.int8)))
        s = OperatorSchema()
        s.AddGeneratedColumns(catalog_of([t])[name], ["k", "s"])
        src = ScanOperator(s, catalog_of([t])[name])
        key = ColRefE(src, "k")
        aggs = [Min(ColRef(src, "s")), Max(ColRef(src, "s")), Count(), Count(ColRef(src, "s"))]
        o = OperatorSchema()
        o.AddDerivedColumn("k", VirtColRef(key, 0))
        for i, a in enumerate(aggs):
            o.AddDerivedColumn(f"a{i}", VirtColRef(a, i + 1))
        plan = OutputOperator(GroupByAggregateOperator(o, src, [key], aggs))
        engine.register_table(t)
        ora = Oracle()
        ora.register_table(t)
        assert compare(engine.execute(plan), ora.execute(plan)) == ""
        engine.set_profiling(True)
        ts = []
        for _ in range(5):
            engine.execute(plan, fetch=False)
            ts.append(sum(x["ms"] for x in engine.last_kernels() if x["tag"] == "group by") * 1e3)
        engine.set_profiling(False)
        us.append(sorted(ts)[2])
    assert us[1] < 10 * us[0]
