"""Queries that outgrow what their block of the engine holds: more tied roots
than frontier slots, path slots reserved past the end of the store, one wall
of tied paths beside other queries, against the oracle.  The overflow is detected, nothing behind the end is read, and the
handle answers other queries afterwards."""
import numpy as np
import pytest

import cpg_b200
import oracle

pytestmark = pytest.mark.gpu


def tied_roots(n_src):
    """n_src sources with one unit edge each into one sink: every path costs 1."""
    src = np.arange(n_src, dtype=np.int32)
    return n_src + 1, src, np.full(n_src, n_src, np.int32), np.ones(n_src, np.float32)


def tied_wall(diamonds):
    """2^diamonds paths of the same cost between one source and one sink."""
    a = 3 * np.arange(diamonds)
    src = np.stack([a, a, a + 1, a + 2], 1).ravel()
    dst = np.stack([a + 1, a + 2, a + 3, a + 3], 1).ravel()
    return (3 * diamonds + 1, src.astype(np.int32), dst.astype(np.int32),
            np.ones(src.size, np.float32))


def generated(seed, n_pins=2000, weight_kind=0):
    d = cpg_b200.generate(cpg_b200.gen_params(
        seed=seed, n_pins=n_pins, n_levels=20, n_first=8, n_last=8, level_span=3, degree_kind=0,
        deg_lo=1, deg_hi=5, weight_kind=weight_kind, iw_lo=1, iw_hi=9, add_virtual=1))
    return d.n, d.src, d.dst, d.w


def expected(graph, k, ref_roots):
    return oracle.OracleGraph.from_edges(*graph).closure_topk(k, ref_roots=ref_roots)[0]["slack"]


def bits_equal(a, b):
    return np.array_equal(np.asarray(a, np.float32).view(np.uint32),
                          np.asarray(b, np.float32).view(np.uint32))


def dag_of(graph):
    n, src, dst, w = graph
    return cpg_b200.Dag(n, src, dst, w)


def run_batch(graphs, gi, ks, root_seeding, engine_ctas=0):
    """Costs of the queries and the batch's statistics."""
    if engine_ctas:
        b = cpg_b200.Batch.__new__(cpg_b200.Batch)
        o = cpg_b200.Options()
        cpg_b200.lib.cpg_options_init(cpg_b200.C.byref(o))
        o.division, o.root_seeding, o.engine_ctas = cpg_b200.DIV_IEEE, root_seeding, engine_ctas
        b._b, b.ks = cpg_b200.C.c_void_p(), []
        assert cpg_b200.lib.cpg_batch_create(cpg_b200.C.byref(b._b), cpg_b200.C.byref(o)) == 0
    else:
        b = cpg_b200.Batch(division=cpg_b200.DIV_IEEE, root_seeding=root_seeding)
    with b:
        for g in graphs:
            b.add_dag(dag_of(g))
        b.commit()
        b.set_queries(gi, ks)
        b.run()
        return [b.costs(q) for q in range(len(ks))], b.stats()


@pytest.mark.parametrize("n_src,k", [(67072, 1), (67073, 1), (100_000, 1), (100_000, 3000),
                                     (150_000, 4096), (150_000, 4097)])
def test_more_tied_roots_than_frontier_slots(n_src, k):
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, root_seeding=cpg_b200.ROOTS_ALL) as g:
        g.load_edges(*tied_roots(n_src))
        g.report_paths(k)
        assert bits_equal(g.get_slacks(k), np.ones(k, np.float32))
        g.load_edges(*generated(5))
        g.report_paths(500)
        assert bits_equal(g.get_slacks(500), expected(generated(5), 500, 0))


def test_tied_roots_of_a_small_query_beside_large_ones():
    graphs = [tied_roots(100_000), generated(6), generated(7, weight_kind=1)]
    gi, ks = [0, 1, 2, 1], [1, 20_000, 16_000, 3]
    got, _ = run_batch(graphs, gi, ks, cpg_b200.ROOTS_ALL)
    want = [expected(g, max(ks), 0) for g in graphs[1:]]
    assert bits_equal(got[0], [1.0])
    for q in (1, 2, 3):
        assert bits_equal(got[q], want[gi[q] - 1][:ks[q]]), q


@pytest.mark.parametrize("queries", [256, 257, 600])
def test_small_queries_of_the_grid_launch_reserve_past_the_path_store(queries):
    # a store of 65,536 slots and the graph's source, which the chunks that the
    # blocks take can fill
    graphs = [generated(8)]
    want = expected(graphs[0], 40, 0)
    ks = [1 + q % 40 if queries == 600 else 1 for q in range(queries)]
    got, _ = run_batch(graphs, [0] * queries, ks, cpg_b200.ROOTS_ALL, engine_ctas=8)
    for q in range(queries):
        assert bits_equal(got[q], want[:ks[q]]), q


def test_wall_of_ties_beside_others_needs_no_rerun():
    # 131,072 tied paths for k = 100: more than 300 times its part of the room
    graphs = [tied_wall(17)] + [generated(20 + i, weight_kind=i % 2) for i in range(3)]
    gi = [0] + [1 + q % 3 for q in range(47)]
    ks = [100] + [4000 - q for q in range(47)]
    got, stats = run_batch(graphs, gi, ks, cpg_b200.ROOTS_REFERENCE)
    want = [expected(g, 4000, 1) for g in graphs[1:]]
    assert bits_equal(got[0], np.full(100, 34.0))
    for q in range(1, 48):
        assert bits_equal(got[q], want[gi[q] - 1][:ks[q]]), q
    assert stats["retries"] == 0


@pytest.mark.parametrize("beside", [20_000, 4000])
def test_wall_of_ties_beside_queries_of_the_grid_launch(beside):
    graphs = [tied_wall(16), generated(30)]
    got, stats = run_batch(graphs, [0, 1, 0, 1, 1], [7, beside, 300, 50, beside - 1],
                           cpg_b200.ROOTS_ALL)
    want = expected(graphs[1], beside, 0)
    assert bits_equal(got[0], np.full(7, 32.0)) and bits_equal(got[2], np.full(300, 32.0))
    for q, k in ((1, beside), (3, 50), (4, beside - 1)):
        assert bits_equal(got[q], want[:k]), q


def test_served_wall_of_ties_needs_no_rerun_and_no_allocation():
    graphs = [tied_wall(17), generated(41), generated(42, weight_kind=1)]
    want = [None] + [expected(g, 4000, 1) for g in graphs[1:]]
    with cpg_b200.Server(division=cpg_b200.DIV_IEEE) as s:
        for g in graphs:
            s.add_dag(dag_of(g))
        s.start()
        asked = [(q % 3, 100 if q % 3 == 0 else 4000 - q) for q in range(60)]
        for (g, k), t in zip(asked, [s.submit(g, k) for g, k in asked]):
            costs = s.wait(t)[0]
            assert bits_equal(costs, np.full(k, 34.0) if g == 0 else want[g][:k]), (g, k)
        stats = s.stats()
    assert stats["retries"] == 0 and stats["loop_allocs"] == 0


@pytest.mark.parametrize("k", [1, 100, 4096, 5000])
@pytest.mark.parametrize("diamonds", [15, 16, 18])
def test_tied_paths_around_what_a_block_walks(diamonds, k):
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE) as g:
        g.load_edges(*tied_wall(diamonds))
        g.report_paths(k)
        nodes = g.get_pfxt_nodes(k)
        assert bits_equal(g.get_slacks(k), np.full(k, 2.0 * diamonds))
        assert bits_equal(nodes["slack"], np.full(k, 2.0 * diamonds))
        v = g.path_vertices(k - 1)
        assert v[0] == 0 and v[-1] == 3 * diamonds and v.size == 2 * diamonds + 1


@pytest.mark.parametrize("n_src", [4097, 65536, 65537, 90_000])
@pytest.mark.parametrize("k", [50, 4096])
def test_many_sources_alone_and_beside_others(n_src, k):
    w = np.random.default_rng(n_src).uniform(1, 100, n_src).astype(np.float32)
    graphs = [tied_roots(n_src)[:3] + (w,), generated(31)]
    want = [expected(graphs[0], k, 0), expected(graphs[1], 700, 0)]
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, root_seeding=cpg_b200.ROOTS_ALL) as g:
        g.load_edges(*graphs[0])
        g.report_paths(k)
        assert bits_equal(g.get_slacks(k), want[0])
        assert g.path_vertices(0).size == 2
    got, _ = run_batch(graphs, [1, 0, 1], [700, k, 20], cpg_b200.ROOTS_ALL)
    assert bits_equal(got[0], want[1]) and bits_equal(got[1], want[0])
    assert bits_equal(got[2], want[1][:20])


@pytest.mark.parametrize("k", [2559, 2560, 2561])
def test_dense_graph_around_the_whole_limit(k):
    d = cpg_b200.generate(cpg_b200.gen_params(
        seed=3, n_pins=1500, n_levels=12, n_first=8, n_last=8, level_span=3, degree_kind=1,
        deg_mean=12.0, deg_cap=40, add_virtual=1))
    assert d.m >= 8 * d.n
    graph = (d.n, d.src, d.dst, d.w)
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE) as g:
        g.load_edges(*graph)
        g.report_paths(k)
        assert bits_equal(g.get_slacks(k), expected(graph, k, 1))


@pytest.mark.parametrize("queries", [2, 5, 8])
def test_few_queries_around_the_whole_limit(queries):
    graphs = [generated(50 + i, weight_kind=i % 2) for i in range(2)]
    line = min(16384, 8192 + 1024 * queries)
    want = [expected(g, line + 3, 0) for g in graphs]
    for least in (line - 1, line, line + 1):
        ks = [least + q % 3 for q in range(queries)]
        got, _ = run_batch(graphs, [q % 2 for q in range(queries)], ks, cpg_b200.ROOTS_ALL)
        for q in range(queries):
            assert bits_equal(got[q], want[q % 2][:ks[q]]), q


def test_served_query_that_needs_more_than_there_is_fails_alone():
    graphs = [tied_wall(20), generated(45)]
    want = expected(graphs[1], 2000, 1)
    try:
        with cpg_b200.Server(division=cpg_b200.DIV_IEEE, hbm_budget_bytes=64 << 20) as s:
            for g in graphs:
                s.add_dag(dag_of(g))
            s.start()
            cpg_b200.debug_fail_allocs_above(4 << 20)   # a million tied paths need more
            with pytest.raises(cpg_b200.CpgError) as e:
                s.wait(s.submit(0, 100))
            assert e.value.status == 3                  # out of memory
            assert bits_equal(s.wait(s.submit(1, 2000))[0], want)
            cpg_b200.debug_fail_allocs_above(0)
            assert bits_equal(s.wait(s.submit(0, 100))[0], np.full(100, 40.0))
    finally:
        cpg_b200.debug_fail_allocs_above(0)
