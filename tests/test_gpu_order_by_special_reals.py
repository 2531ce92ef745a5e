"""ORDER BY over REAL keys that hold both zeros, infinities and NaN, at sizes
of every sort (all pairs of rows, key ranges, radix passes)."""

import numpy as np
import pytest

from kushdb_b200.data import HostColumn, HostTable, catalog_of
from kushdb_b200.plan import ColRef, OperatorSchema, OrderByOperator, OutputOperator, ScanOperator, Type
from parity import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def _table(name, n, nan, nulls):
    rng = np.random.default_rng(n)
    special = [0.0, -0.0, np.inf, -np.inf, 1.5, -1.5, 5e-324, -5e-324]
    if nan:
        special += [np.nan, -np.nan]
    k = np.where(rng.random(n) < 0.5, rng.choice(special, n), rng.normal(0, 1, n))
    t = HostTable(name)
    t.add(HostColumn("id", Type.Int(), values=np.arange(n, dtype=np.int32)))
    t.add(HostColumn("k", Type.Real(), values=k, nulls=(rng.random(n) < 0.1).astype(np.int8) if nulls else None))
    t.add(HostColumn("g", Type.Real(), values=rng.integers(0, 3, n).astype(np.float64)))
    return t


def _plan(t, keys, asc):
    rel = catalog_of([t])[t.name]
    s = OperatorSchema()
    s.AddGeneratedColumns(rel, ["id", "k", "g"])
    base = ScanOperator(s, rel)
    out = OperatorSchema()
    out.AddPassthroughColumns(base)
    return OutputOperator(OrderByOperator(out, base, [ColRef(base, k) for k in keys], asc))


SIZES = [2, 40, 1000, 2048, 2049, 3000, 4097, 20_000]


# -0.0 equals 0.0: such rows come in the tie order
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("keys,asc,nulls", [(["k"], [True], False), (["k"], [False], False), (["k"], [True], True),
                                            (["g", "k"], [True, False], False)])
def test_zeros_and_infinities_match_oracle(engine, n, keys, asc, nulls):
    from oracle import Oracle
    t = _table(f"z{n}{len(keys)}{asc[0]}{nulls}", n, False, nulls)
    engine.register_table(t)
    o = Oracle()
    o.register_table(t)
    plan = _plan(t, keys, asc)
    assert compare(engine.execute(plan), o.execute(plan)) == ""


# every row comes back once; numbers ascend, with the NaNs of either sign at their ends
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("keys,asc,nulls", [(["k"], [True], False), (["k"], [False], False), (["k"], [False], True),
                                            (["g", "k"], [True, False], False)])
def test_nan_keys_lose_no_row(engine, n, keys, asc, nulls):
    t = _table(f"n{n}{len(keys)}{asc[0]}{nulls}", n, True, nulls)
    engine.register_table(t)
    ids = np.asarray(engine.execute(_plan(t, keys, asc)).columns[0].values)
    assert np.array_equal(np.sort(ids), np.arange(n))
    k = t.columns["k"].values[ids]
    bits = np.where(k == 0.0, 0.0, k).view(np.int64)
    rank = np.where(bits < 0, ~bits ^ np.int64(-2**63), bits)
    null = np.zeros(n, bool) if not nulls else t.columns["k"].nulls[ids] != 0
    g = t.columns["g"].values[ids] if len(keys) > 1 else np.zeros(n)
    if not asc[-1]:
        rank = ~rank
    place = [(a, b if asc[-1] else not b, 0 if b else c) for a, b, c in zip(g.tolist(), null.tolist(), rank.tolist())]
    assert place == sorted(place)


# kdb_sort: the same order, ties in input order
@pytest.mark.parametrize("n", [40, 2049, 20_000])
@pytest.mark.parametrize("asc", [True, False])
def test_sort_rows_of_zeros_and_infinities(engine, n, asc):
    from kushdb_b200.operators import sort_rows
    t = _table(f"sr{n}{asc}", n, False, False)
    engine.register_table(t)
    k = t.columns["k"].values + 0.0  # one zero
    want = np.argsort(k if asc else -k, kind="stable")
    assert np.array_equal(sort_rows(engine, t.name, ["k"], [asc]).rows(), want)
