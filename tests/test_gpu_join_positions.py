"""The order of rows and groups that come out of joins (a row's place is its
probe row's, then its build row's): several joins above one another, and more
probe rows than 24 bits count."""

import numpy as np
import pytest

from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.plan import (ColRef, ColRefE, Count, GroupByAggregateOperator, HashJoinOperator, OperatorSchema,
                              OrderByOperator, OutputOperator, ScanOperator, Type, VirtColRef)
from parity import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _scan(t):
    s = OperatorSchema()
    s.AddGeneratedColumns(catalog_of([t])[t.name], list(t.columns))
    return ScanOperator(s, catalog_of([t])[t.name])


def _ints(name, **cols):
    t = HostTable(name)
    for c, v in cols.items():
        nulls = None
        if isinstance(v, tuple):
            v, nulls = v
        t.add(HostColumn(c, Type.Int(), values=np.asarray(v, np.int32), nulls=nulls))
    return t


def _groups(src, key, nullable=None):
    k = ColRefE(src, key)
    aggs = [Count()] + ([Count(ColRef(src, nullable))] if nullable else [])
    o = OperatorSchema()
    o.AddDerivedColumn("k", VirtColRef(k, 0))
    for i, a in enumerate(aggs):
        o.AddDerivedColumn(f"n{i}", VirtColRef(a, 1 + i))
    return OutputOperator(GroupByAggregateOperator(o, src, [k], aggs))


# first table's rows probe the second, the pairs probe the third (each with several rows per key)
@pytest.mark.parametrize("levels", [1, 2, 3])
@pytest.mark.parametrize("ordered", [False, True])
def test_order_of_nested_joins_matches_oracle(engine, levels, ordered):
    from oracle import Oracle
    rng = np.random.default_rng(levels)
    n = 5003
    fact = _ints(f"np{levels}{ordered}", a=rng.integers(0, 300, n), b=rng.integers(0, 40, n), c=rng.integers(0, 25, n),
                 g=rng.integers(0, 700, n), x=(rng.integers(0, 9, n), (rng.random(n) < 0.3).astype(np.int8)))
    o = Oracle()
    engine.register_table(fact)
    o.register_table(fact)
    src, keep = _scan(fact), ["a", "b", "c", "g", "x"]
    for level, key in list(enumerate("abc"))[:levels]:
        m = (300, 40, 25)[level]
        dim = _ints(f"nd{levels}{ordered}{level}", k=rng.permutation(2 * m) % m, h=rng.integers(0, 5, 2 * m))
        engine.register_table(dim)
        o.register_table(dim)
        d = _scan(dim)
        js = OperatorSchema()
        js.AddPassthroughColumns(src, keep, 1)
        src = HashJoinOperator(js, d, src, [ColRef(d, "k", 0)], [ColRef(src, key, 1)])
    if ordered:  # ties of the sort key come in the tie order of the stream
        out = OperatorSchema()
        out.AddPassthroughColumns(src)
        plan = OutputOperator(OrderByOperator(out, src, [ColRef(src, "b")], [True]))
    else:
        plan = _groups(src, "g", "x")
    assert compare(engine.execute(plan), o.execute(plan)) == ""


def test_groups_of_more_than_2_24_probe_rows(engine):
    n, m = (1 << 24) + 700_001, 1003
    rng = np.random.default_rng(6)
    fk = rng.integers(0, m - 3, n)
    fk[[5, n - 2, n - 1]] = m - 1, m - 2, m - 3
    fact, dim = _ints("wide_fact", k=fk), _ints("wide_dim", k=np.arange(m), g=rng.permutation(m))
    engine.register_table(fact)
    engine.register_table(dim)
    d, f = _scan(dim), _scan(fact)
    js = OperatorSchema()
    js.AddPassthroughColumns(d, ["k", "g"], 0)
    j = HashJoinOperator(js, d, f, [ColRef(d, "k", 0)], [ColRef(f, "k", 1)])
    keys, first = np.unique(fk, return_index=True)
    want = keys[np.argsort(first)]
    for key, of in (("k", want), ("g", dim.columns["g"].values[want])):
        r = engine.execute(_groups(j, key))
        assert np.array_equal(r.columns[0].values, of)
        assert np.array_equal(r.columns[1].values, np.bincount(fk)[want])
    engine.drop_table("wide_fact")
