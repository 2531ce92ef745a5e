"""Batched form: many uneven scan-select -> hash-join -> group-by queries in
one captured CUDA graph.  Every query's batched result must equal the plain
executor's result for the same plan (same groups in the same first-
occurrence order; sums within 1e-12 relative), and the oracle's for a few."""

import numpy as np
import pytest

from kushdb_b200 import workloads as wl
from parity import REL_TOL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    from kushdb_b200.engine import Batch, Engine
    e = Engine(0)
    qs = wl.batch_tables(n_queries=48, min_fact=100, max_fact=200_000, seed=3, prefix="tb")
    for d, f, _, _ in qs:
        e.register_table(d)
        e.register_table(f)
    b = Batch(e, [wl.batch_query_desc(*q) for q in qs])
    yield e, b, qs
    b.close()
    e.close()


def _check_against_plain(e, b, qs):
    b.run()
    for i, q in enumerate(qs):
        keys, sums = b.result(i)
        plain = e.execute(wl.batch_plan(*q))
        pk = np.asarray(plain.columns[0].values)
        ps = np.asarray(plain.columns[1].values)
        assert np.array_equal(keys, pk), f"query {i}: keys differ"
        assert np.all(np.abs(sums - ps) <= REL_TOL * np.maximum(np.abs(ps), 1e-300)), f"query {i}: sums"


@pytest.mark.parametrize("block,lf,fanout", [(256, 0.5, 1), (128, 0.9, 64), (512, 0.7, 1024)])
def test_batch_matches_plain_executor(setup, block, lf, fanout):
    e, b, qs = setup
    b.configure(block, lf, fanout)
    _check_against_plain(e, b, qs)


def test_batch_matches_oracle(setup):
    from oracle import Oracle
    e, b, qs = setup
    b.configure()
    b.run()
    for i in (0, 7, 23):
        o = Oracle()
        o.register_table(qs[i][0])
        o.register_table(qs[i][1])
        ref = o.execute(wl.batch_plan(*qs[i]))
        keys, sums = b.result(i)
        assert np.array_equal(keys, np.asarray(ref.columns[0].values))
        rs = np.asarray(ref.columns[1].values)
        assert np.all(np.abs(sums - rs) <= REL_TOL * np.maximum(np.abs(rs), 1e-300))


def test_autotuner_picks_a_timed_configuration(setup):
    e, b, qs = setup
    report = b.tune(reps=1)
    assert len(report) == 3 * 3 * 4
    best = min(report, key=lambda r: r["ms"])
    cfg = b.config()
    assert (cfg["block"], cfg["fanout"]) == (best["block"], best["fanout"])
    assert abs(cfg["load_factor"] - best["load_factor"]) < 1e-9
    _check_against_plain(e, b, qs)


def test_batch_rejects_non_unique_dimension_keys():
    from kushdb_b200.data import HostColumn
    from kushdb_b200.engine import Batch, Engine, KdbError
    e = Engine(0)
    (d, f, lt, seg), = wl.batch_tables(n_queries=1, min_fact=1000, max_fact=1000, seed=9, prefix="dup")
    d.columns["d_key"] = HostColumn("d_key", wl.Type.Int(), values=np.zeros(d.rows, np.int32))
    e.register_table(d)
    e.register_table(f)
    b = Batch(e, [wl.batch_query_desc(d, f, lt + 10_000, seg)])
    with pytest.raises(KdbError):
        b.run()
    b.close()
    e.close()


# the group order's edges: one bitmap word (32 fact rows), one order chunk
# (32768 fact rows), several chunks with a partial last one
@pytest.mark.parametrize("facts", [1, 31, 32, 33, 32_767, 32_768, 32_769, 65_537, 300_001])
def test_batch_group_order_at_bitmap_edges(facts):
    from kushdb_b200.engine import Batch, Engine
    with Engine(0) as e:
        qs = [wl.batch_tables(n_queries=1, min_fact=n + 0.5, max_fact=n + 0.5, seed=n, prefix=f"be{i}_")[0]
              for i, n in enumerate((facts, 1000, facts))]
        for d, f, _, _ in qs:
            e.register_table(d)
            e.register_table(f)
        b = Batch(e, [wl.batch_query_desc(*q) for q in qs])
        _check_against_plain(e, b, qs)
        _check_against_plain(e, b, qs)  # a second run of the same graph
        b.close()


# more order chunks (of 32768 fact rows) than a block counts in shared memory (1024)
def test_batch_group_order_beyond_the_shared_counters():
    from kushdb_b200.data import HostColumn, HostTable
    from kushdb_b200.engine import Batch, Engine
    nf, nd = 1025 * 32_768 + 77, 1003
    rng = np.random.default_rng(8)
    d, f = HostTable("bl_dim"), HostTable("bl_fact")
    d.add(HostColumn("d_key", wl.Type.Int(), values=(np.arange(nd) * 7).astype(np.int32)))
    d.add(HostColumn("d_date", wl.Type.Date(), values=rng.integers(2440588, 2450000, nd).astype(np.int32)))
    d.add(HostColumn("d_seg", wl.Type.Int(), values=np.zeros(nd, np.int32)))
    fk = rng.integers(0, nd - 3, nf)
    fk[[5, nf - 2, nf - 1]] = nd - 1, nd - 2, nd - 3  # groups whose first rows lie in the first and the last chunk
    f.add(HostColumn("f_fk", wl.Type.Int(), values=(fk * 7).astype(np.int32)))
    f.add(HostColumn("f_price", wl.Type.Real(), values=rng.random(nf)))
    f.add(HostColumn("f_disc", wl.Type.Real(), values=rng.integers(0, 10, nf) / 100.0))
    with Engine(0) as e:
        e.register_table(d)
        e.register_table(f)
        q = (d, f, 2449000, 0)
        b = Batch(e, [wl.batch_query_desc(*q)])
        _check_against_plain(e, b, [q])
        b.close()
