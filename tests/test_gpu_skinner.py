"""Skinner multiway joins (JOB-style star and chain shapes, Zipf-skewed
foreign keys, LIKE '%tok%' filters) against the oracle: the adaptive
episode engine must return exactly the join's result for every budget."""

import pytest

from kushdb_b200 import workloads as wl
from parity import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from kushdb_b200.engine import Engine
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("shape,n_tables,zipf", [("star", 6, 0.0), ("chain", 6, 0.0), ("star", 8, 1.5),
                                                 ("chain", 7, 1.5)])
@pytest.mark.parametrize("budget", [2000, 1 << 20])
def test_skinner_multiway_matches_oracle(engine, shape, n_tables, zipf, budget):
    from oracle import Oracle
    tables, tokens = wl.skinner_tables(shape, n_tables, min_rows=1000, max_rows=20_000, zipf_s=zipf,
                                       seed=11 + n_tables, prefix=f"{shape}{n_tables}{int(zipf)}_")
    plan = wl.skinner_plan(tables, tokens, shape)
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    engine.set_skinner(budget, seed=1)
    try:
        g = engine.execute(plan)
    finally:
        engine.set_skinner()
    ref = o.execute(plan)
    assert compare(g, ref) == ""
    assert engine.last_skinner_episodes() >= 1


def test_aggregate_fused_into_episodes_matches_materialised(engine):
    """COUNT/MIN over the join evaluated inside the episode kernel equals the
    same aggregate over the materialised join result."""
    tables, tokens = wl.skinner_tables("chain", 6, min_rows=1000, max_rows=30_000, zipf_s=1.5, seed=77,
                                       prefix="fuse_")
    for t in tables:
        engine.register_table(t)
    plan = wl.skinner_plan(tables, tokens, "chain").to_json()
    engine.set_skinner(5000, seed=3)
    try:
        fused = engine.execute(plan)
        engine.set_option("KDB_NO_SKINNER_AGG", "1")
        try:
            plain = engine.execute(plan)
        finally:
            engine.set_option("KDB_NO_SKINNER_AGG", None)
    finally:
        engine.set_skinner()
    assert compare(fused, plain) == ""


@pytest.mark.parametrize("split,tasks", [(8, 1 << 16), (8, 16), (64, 1 << 16)])
@pytest.mark.parametrize("shape,n_tables", [("chain", 7), ("star", 8)])
@pytest.mark.parametrize("fused", [True, False])
def test_hot_runs_as_tasks_match_oracle(engine, split, tasks, shape, n_tables, fused):
    """Runs longer than `split` candidates at position 3 and deeper go to the
    task queues (a queue of `tasks` entries: with 16 it fills, and the rest
    is walked in place); the result stays exactly the join's."""
    from oracle import Oracle
    tables, tokens = wl.skinner_tables(shape, n_tables, min_rows=1000, max_rows=20_000, zipf_s=1.5,
                                       seed=31 + n_tables, prefix=f"hot{shape}{n_tables}_")
    plan = wl.skinner_plan(tables, tokens, shape)
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    engine.set_option("KDB_SKINNER_SPLIT", str(split))
    engine.set_option("KDB_SKINNER_TASKS", str(tasks))
    if not fused:  # results materialised (slot allocation, regrowth) instead of folded
        engine.set_option("KDB_NO_SKINNER_AGG", "1")
    engine.set_skinner(3000, seed=2)
    try:
        g = engine.execute(plan)
    finally:
        for k in ("KDB_SKINNER_SPLIT", "KDB_SKINNER_TASKS", "KDB_NO_SKINNER_AGG"):
            engine.set_option(k, None)
        engine.set_skinner()
    assert compare(g, o.execute(plan)) == ""


@pytest.mark.parametrize("batch", [1, 4, 16])
@pytest.mark.parametrize("policy", ["uct", "random"])
def test_episode_batches_keep_the_result(engine, batch, policy):
    """Episodes run in batches (several join orders per launch, rewards
    corrected after the batch): the result is the join's for every batch
    size, and with more than one episode per batch there are fewer batches
    than episodes."""
    from oracle import Oracle
    tables, tokens = wl.skinner_tables("chain", 7, min_rows=2000, max_rows=40_000, zipf_s=1.5, seed=91,
                                       prefix=f"batch{batch}{policy}_")
    plan = wl.skinner_plan(tables, tokens, "chain", like_tables=(2,))
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    engine.set_option("KDB_SKINNER_BATCH", str(batch))
    engine.set_skinner_policy(policy)
    engine.set_skinner(2000, seed=4)
    try:
        g = engine.execute(plan)
        episodes, batches = engine.last_skinner_episodes(), engine.last_skinner_batches()
    finally:
        engine.set_option("KDB_SKINNER_BATCH", None)
        engine.set_skinner_policy("uct")
        engine.set_skinner()
    assert compare(g, o.execute(plan)) == ""
    assert episodes >= batches >= 1
    if batch == 1:
        assert batches == episodes
    elif episodes > 4 * batch:
        assert batches < episodes


# the grouped indexes' edges: one row, a CTA's rows (1024) and one more or
# less, several CTAs; unique keys, few keys, one key for every row, NULL keys
@pytest.mark.parametrize("rows", [1, 2, 1023, 1024, 1025, 40_003])
@pytest.mark.parametrize("keys", ["unique", "few", "one", "null"])
def test_grouped_index_edges_match_oracle(engine, rows, keys):
    import numpy as np
    from kushdb_b200.data import HostColumn, HostTable, catalog_of
    from kushdb_b200.plan import (AggregateOperator, ColRef, Count, Eq, Max, OperatorSchema, OutputOperator,
                                  ScanOperator, SkinnerJoinOperator, Sum, Type, VirtColRef)
    from oracle import Oracle
    rng = np.random.default_rng(rows)
    n_b = 700
    k = {"unique": rng.permutation(rows), "few": rng.integers(0, 5, rows), "one": np.full(rows, 3),
         "null": rng.integers(0, 50, rows)}[keys].astype(np.int32)
    nulls = (rng.random(rows) < 0.5).astype(np.int8) if keys == "null" else None
    a = HostTable(f"ix_a_{rows}_{keys}")
    a.add(HostColumn("k", Type.Int(), values=k, nulls=nulls))
    a.add(HostColumn("v", Type.Int(), values=rng.integers(0, 1000, rows).astype(np.int32)))
    b = HostTable(f"ix_b_{rows}_{keys}")
    b.add(HostColumn("k", Type.Int(), values=rng.integers(0, 60, n_b).astype(np.int32)))
    b.add(HostColumn("g", Type.BigInt(), values=rng.integers(0, 20, n_b)))
    c = HostTable(f"ix_c_{rows}_{keys}")
    c.add(HostColumn("g", Type.BigInt(), values=np.arange(25)))
    tables = [a, b, c]
    db = catalog_of(tables)
    scans = []
    for t in tables:
        s = OperatorSchema()
        s.AddGeneratedColumns(db[t.name], list(t.columns))
        scans.append(ScanOperator(s, db[t.name]))
    js = OperatorSchema()
    js.AddPassthroughColumns(scans[0], ["v"], 0)
    js.AddPassthroughColumns(scans[2], ["g"], 2)
    join = SkinnerJoinOperator(js, scans, [Eq(ColRef(scans[0], "k", 0), ColRef(scans[1], "k", 1)),
                                           Eq(ColRef(scans[1], "g", 1), ColRef(scans[2], "g", 2))])
    aggs = [Count(), Sum(ColRef(join, "v")), Max(ColRef(join, "g"))]
    out = OperatorSchema()
    for i, name in enumerate(("n", "total", "most")):
        out.AddDerivedColumn(name, VirtColRef(aggs[i], i))
    plan = OutputOperator(AggregateOperator(out, join, aggs))
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    engine.set_skinner(5000, seed=1)
    try:
        g = engine.execute(plan)
    finally:
        engine.set_skinner()
    assert compare(g, o.execute(plan)) == ""


# filtered children are counted while the others' indexes build: none, some or
# all of them filtered, a filter that keeps one row, all rows or none
@pytest.mark.parametrize("filtered", [(), (1,), (0, 2), (0, 1, 2)])
@pytest.mark.parametrize("keep", ["none", "one", "some", "all"])
def test_filtered_children_match_oracle(engine, filtered, keep):
    import numpy as np
    from kushdb_b200.data import HostColumn, HostTable, catalog_of
    from kushdb_b200.plan import (AggregateOperator, ColRef, Count, Eq, Literal, Lt, OperatorSchema, OutputOperator,
                                  ScanOperator, ScanSelectOperator, SkinnerJoinOperator, Sum, Type, VirtColRef)
    from oracle import Oracle
    rng = np.random.default_rng(17)
    tables = []
    for i, n in enumerate((3000, 400, 1500)):
        t = HostTable(f"fc_{i}_{len(filtered)}_{keep}")
        t.add(HostColumn("k", Type.Int(), values=rng.integers(0, 90, n).astype(np.int32)))
        t.add(HostColumn("g", Type.Int(), values=rng.integers(0, 120, n).astype(np.int32),
                         nulls=(rng.random(n) < 0.1).astype(np.int8)))
        t.add(HostColumn("id", Type.Int(), values=np.arange(n, dtype=np.int32)))
        tables.append(t)
    below = {"none": 0, "one": 1, "some": 350, "all": 3000}[keep]
    db = catalog_of(tables)
    kids = []
    for i, t in enumerate(tables):
        s = OperatorSchema()
        s.AddGeneratedColumns(db[t.name], ["k", "g", "id"])
        if i in filtered:
            out = OperatorSchema()
            out.AddVirtualPassthroughColumns(s, ["k", "g", "id"])
            kids.append(ScanSelectOperator(out, s, db[t.name], [Lt(VirtColRef(s, "id"), Literal(below))]))
        else:
            kids.append(ScanOperator(s, db[t.name]))
    js = OperatorSchema()
    js.AddPassthroughColumns(kids[0], ["id"], 0)
    join = SkinnerJoinOperator(js, kids, [Eq(ColRef(kids[0], "k", 0), ColRef(kids[1], "k", 1)),
                                          Eq(ColRef(kids[1], "g", 1), ColRef(kids[2], "g", 2))])
    aggs = [Count(), Sum(ColRef(join, "id"))]
    out = OperatorSchema()
    for i, name in enumerate(("n", "total")):
        out.AddDerivedColumn(name, VirtColRef(aggs[i], i))
    plan = OutputOperator(AggregateOperator(out, join, aggs))
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    want = o.execute(plan)
    for _ in range(2):
        assert compare(engine.execute(plan), want) == ""


# the index hashes by the key column's stored type; lookups hash the same way
@pytest.mark.parametrize("kind", ["BOOLEAN", "SMALLINT", "INT", "DATE", "BIGINT", "REAL", "TEXT"])
def test_index_key_types_match_oracle(engine, kind):
    import numpy as np
    from kushdb_b200.data import HostColumn, HostTable, catalog_of
    from kushdb_b200.plan import (AggregateOperator, ColRef, Count, Eq, OperatorSchema, OutputOperator, ScanOperator,
                                  SkinnerJoinOperator, Sum, Type, VirtColRef)
    from oracle import Oracle
    rng = np.random.default_rng(29)
    tables = []
    for i, n in enumerate((900, 300, 60)):
        t = HostTable(f"kt_{kind}_{i}")
        v = rng.integers(-20, 20, n)
        nulls = (rng.random(n) < 0.1).astype(np.int8)
        if kind == "TEXT":
            t.add(HostColumn.from_strings("k", ["s" * (int(x) % 5 + 5) + str(int(x)) for x in v], nulls))
        else:
            values = {"BOOLEAN": (v > 15).astype(np.int8), "SMALLINT": v.astype(np.int16), "INT": v.astype(np.int32),
                      "DATE": (v + 2440588).astype(np.int32), "BIGINT": v * (1 << 33),
                      "REAL": np.where(v == 0, -0.0 if i else 0.0, v * 0.37)}[kind]
            t.add(HostColumn("k", Type(kind), values=values, nulls=nulls))
        t.add(HostColumn("g", Type.Int(), values=rng.integers(0, 40, n).astype(np.int32)))
        tables.append(t)
    db = catalog_of(tables)
    scans = []
    for t in tables:
        s = OperatorSchema()
        s.AddGeneratedColumns(db[t.name], ["k", "g"])
        scans.append(ScanOperator(s, db[t.name]))
    js = OperatorSchema()
    js.AddPassthroughColumns(scans[0], ["g"], 0)
    join = SkinnerJoinOperator(js, scans, [Eq(ColRef(scans[0], "k", 0), ColRef(scans[1], "k", 1)),
                                           Eq(ColRef(scans[1], "g", 1), ColRef(scans[2], "g", 2))])
    aggs = [Count(), Sum(ColRef(join, "g"))]
    out = OperatorSchema()
    for i, name in enumerate(("n", "total")):
        out.AddDerivedColumn(name, VirtColRef(aggs[i], i))
    plan = OutputOperator(AggregateOperator(out, join, aggs))
    o = Oracle()
    for t in tables:
        engine.register_table(t)
        o.register_table(t)
    assert compare(engine.execute(plan), o.execute(plan)) == ""


# a join of 8 tables of at most 1000 rows, in a process of its own: the fixed
# scratch (34 MB of slices and items, the pool's granularity, the kernels) and
# queues as large as such tables need; with room for 2^18 tasks they alone took 50 MB
def test_small_join_takes_little_device_memory():
    import os
    import subprocess
    import sys
    code = (
        "import torch\n"
        "from kushdb_b200 import workloads as wl\n"
        "from kushdb_b200.engine import Engine\n"
        "e = Engine(0)\n"
        "tables, tokens = wl.skinner_tables('chain', 8, 300, 1000, 0.0, prefix='sm')\n"
        "for t in tables: e.register_table(t)\n"
        "plan = wl.skinner_plan(tables, tokens, 'chain').to_json().encode()\n"
        "free = torch.cuda.mem_get_info()[0]\n"
        "e.execute(plan)\n"
        "print((free - torch.cuda.mem_get_info()[0]) >> 20)\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root)
    assert out.returncode == 0, out.stderr[-2000:]
    assert int(out.stdout) <= 96
