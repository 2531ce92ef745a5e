"""Results that several host threads copy (16 MB and more), that get an array
per column (more than 24 MiB), and ORDER BY over more rows than the smallest
number of key ranges serves; results written straight to host memory."""

import ctypes

import numpy as np
import pytest

from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.plan import (AggregateOperator, Avg, ColRef, ColRefE, Count, GroupByAggregateOperator, Lt, Max, Min,
                              OperatorSchema, OrderByOperator, OutputOperator, ScanOperator, SelectOperator, Sum, Type,
                              VirtColRef)

pytestmark = pytest.mark.gpu

COLUMNS = ["id", "s", "b", "t", "r", "d", "nr"]


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _table(name, n):
    rng = np.random.default_rng(n)

    def nulls():
        return (rng.random(n) < 0.2).astype(np.int8)

    t = HostTable(name)
    t.add(HostColumn("id", Type.Int(), values=np.arange(n, dtype=np.int32)))
    t.add(HostColumn("s", Type.SmallInt(), values=rng.integers(-300, 300, n).astype(np.int16), nulls=nulls()))
    t.add(HostColumn("b", Type.Boolean(), values=rng.integers(0, 2, n).astype(np.int8), nulls=nulls()))
    t.add(HostColumn.from_strings("t", ["" if x == 0 else "t%d" % x for x in rng.integers(0, 50, n)], nulls()))
    t.add(HostColumn("r", Type.Real(), values=rng.permutation(n) * 0.37 - 1000.0))
    t.add(HostColumn("d", Type.Date(), values=rng.integers(2440588, 2441600, n).astype(np.int32)))
    t.add(HostColumn("nr", Type.Real(), values=rng.normal(0, 1, n), nulls=nulls()))
    return t


def _order(t, columns, key, asc):
    rel = catalog_of([t])[t.name]
    s = OperatorSchema()
    s.AddGeneratedColumns(rel, list(dict.fromkeys(columns + [key])))
    base = ScanOperator(s, rel)
    out = OperatorSchema()
    out.AddPassthroughColumns(base)
    return OutputOperator(OrderByOperator(out, base, [ColRef(base, key)], [asc]))


def _same_columns(got, want):
    assert got.num_rows == want.num_rows and len(got.columns) == len(want.columns)
    for x, y in zip(got.columns, want.columns):
        assert x.type.to_json() == y.type.to_json() and np.array_equal(x.nulls, y.nulls)
        live = np.asarray(y.nulls) == 0
        if x.type.type_id == "TEXT":
            assert all(a == b for a, b, l in zip(x.values, y.values, live) if l)
        else:
            assert np.array_equal(np.asarray(x.values)[live], np.asarray(y.values)[live])


# 9 bytes per value: one column of 100k rows 0.9 MB, 7 of 300k 18.9 MB, 7 of 500k 31.5 MB; the rows are
# no multiple of a copied piece (16384) and, from 65537 on, more than 4 per range of the smallest sort
@pytest.mark.parametrize("n", [100_003, 300_007, 500_009])
@pytest.mark.parametrize("key,asc", [("r", True), ("d", False), ("nr", True), ("nr", False), ("s", True)])
def test_large_ordered_results_match_oracle(engine, n, key, asc):
    from oracle import Oracle
    t = _table(f"lr{n}", n)
    engine.register_table(t)
    o = Oracle()
    o.register_table(t)
    plan = _order(t, COLUMNS if key == "r" else ["id", "nr", "s"], key, asc)
    _same_columns(engine.execute(plan), o.execute(plan))


@pytest.mark.parametrize("n", [1, 100_003, 300_007, 500_009])
def test_read_at_once_equals_the_column_calls(engine, n):
    t = _table(f"rc{n}", n)
    engine.register_table(t)
    rel = catalog_of([t])[t.name]
    s = OperatorSchema()
    s.AddGeneratedColumns(rel, COLUMNS)
    r = engine.execute(OutputOperator(ScanOperator(s, rel)))
    lib, _, _, handle = r._src
    for c, col in enumerate(r.columns):
        nulls = np.empty(n, np.int8)
        lib.kdb_result_get_nulls(handle, c, nulls.ctypes.data_as(ctypes.c_void_p))
        assert np.array_equal(nulls, col.nulls)
        if col.type.type_id == "TEXT":
            continue
        real = col.type.type_id == "REAL"
        v = np.empty(n, np.float64 if real else np.int64)
        get = lib.kdb_result_get_f64 if real else lib.kdb_result_get_i64
        get(handle, c, v.ctypes.data_as(ctypes.c_void_p))
        assert v.dtype == col.values.dtype and np.array_equal(v, col.values)
        # (a scan's rows come in any order)
        own = t.columns[COLUMNS[c]].nulls
        assert np.array_equal(np.zeros(n, np.int8) if own is None else own[r.columns[0].values], col.nulls)


def _aggregates(t, grouped, empty):
    rel = catalog_of([t])[t.name]
    s = OperatorSchema()
    s.AddGeneratedColumns(rel, COLUMNS)
    src = ScanOperator(s, rel)
    if empty:
        f = OperatorSchema()
        f.AddPassthroughColumns(src)
        src = SelectOperator(f, src, Lt(ColRef(src, "id"), ColRef(src, "id")))
    aggs = [Count(), Sum(ColRef(src, "nr")), Min(ColRef(src, "d")), Max(ColRef(src, "s")), Avg(ColRef(src, "r")),
            Count(ColRef(src, "s"))]
    out = OperatorSchema()
    keys = [ColRefE(src, "b")] if grouped else []
    for i, k in enumerate(keys):
        out.AddDerivedColumn("k", VirtColRef(k, i))
    for i, a in enumerate(aggs):
        out.AddDerivedColumn(f"a{i}", VirtColRef(a, i + len(keys)))
    return OutputOperator(GroupByAggregateOperator(out, src, keys, aggs) if grouped else AggregateOperator(out, src, aggs))


# results in a mapped block, and without one (as when all blocks are taken): the
# same values and NULLs, also of no rows, and kept results stay as they were
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("empty", [False, True])
def test_mapped_results_equal_downloaded_ones(engine, grouped, empty):
    t = _table(f"mr{grouped}{empty}", 20_011)
    engine.register_table(t)
    plan = _aggregates(t, grouped, empty).to_json()
    kept = [engine.execute(plan) for _ in range(4)]  # fresh, recorded, replayed
    engine.set_option("KDB_NO_MAPPED_RESULT", "1")
    try:
        plain = [engine.execute(plan) for _ in range(4)]
    finally:
        engine.set_option("KDB_NO_MAPPED_RESULT", None)
    for r in kept + plain:
        _same_columns(r, plain[0])
    assert plain[0].num_rows == (0 if grouped and empty else 3 if grouped else 1)
