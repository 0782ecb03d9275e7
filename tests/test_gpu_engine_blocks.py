"""Queries on blocks of their own: answered whole up to the edge of the sort
buffer, left to the grid launch beyond it, many in one launch, with piles that
spill out of shared memory, ties, several sources and fewer paths than asked
for, against the oracle and the host-stepped path."""
import numpy as np
import pytest

import cases
import cpg_b200
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 63, 64, 65, 1023, 2048, 4095, 4096, 4097])
@pytest.mark.parametrize("name", ["single20k_f32", "small_int_s13", "tv80_unit_wgts"])
def test_single_query_around_the_whole_limit(name, k):
    n, src, dst, w = cases.load_case(name)
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, root_seeding=cpg_b200.ROOTS_ALL) as g:
        g.load_edges(n, src, dst, w)
        g.report_paths(k)
        got, nodes = g.get_slacks(k), g.get_pfxt_nodes(k)
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, root_seeding=cpg_b200.ROOTS_ALL,
                        host_stepped=True) as g:
        g.load_edges(n, src, dst, w)
        g.report_paths(k)
        want = g.get_slacks(k)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(nodes["slack"].view(np.uint32), want.view(np.uint32))
    par = nodes["parent"]
    assert (par < nodes.size).all() and (nodes["level"][par[par >= 0]] + 1 == nodes["level"][par >= 0]).all()


@pytest.mark.parametrize("queries", [1, 3, 40, 200])
def test_batch_of_whole_and_grid_queries_equals_oracle(queries):
    dags, want = [], []
    ks = [1, 100, 16384, 16385, 5, 0, 30000, 4097]
    for i in range(4):
        dags.append(cpg_b200.generate(cpg_b200.gen_params(
            seed=90 + i, n_pins=400 * (i + 1), n_levels=6 + 4 * i, n_first=4, n_last=4, level_span=2,
            degree_kind=0, deg_lo=1, deg_hi=3 + i, weight_kind=i % 2, iw_lo=1, iw_hi=9,
            add_virtual=int(i != 2))))
        og = oracle.OracleGraph.from_edges(dags[-1].n, dags[-1].src, dags[-1].dst, dags[-1].w)
        want.append(og.closure_topk(max(ks), ref_roots=1)[0]["slack"])
    rng = np.random.default_rng(queries)
    gi = rng.integers(0, 4, queries).tolist()
    kq = [ks[(i + queries) % len(ks)] for i in range(queries)]
    with cpg_b200.Batch(division=cpg_b200.DIV_IEEE) as b:
        for d in dags:
            b.add_dag(d)
        b.commit()
        b.set_queries(gi, kq)
        for rebuild in (True, False):
            b.run(rebuild)
            for q in range(queries):
                x = want[gi[q]][:kq[q]]
                got = b.costs(q)
                assert np.array_equal(got.view(np.uint32), x.view(np.uint32)), (q, gi[q], kq[q])
