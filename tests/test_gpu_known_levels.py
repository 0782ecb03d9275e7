"""Suffix-tree rebuilds over known levels after delay updates: the walk of the
level order from a changed level on (heaps appended), of the whole order, with
and without the heap phase, and of several changed side-by-side graphs, against
the oracle and fresh builds; edge ids out of range change nothing."""
import ctypes as C

import numpy as np
import pytest

import cases
import cpg_b200
import oracle

pytestmark = pytest.mark.gpu


def _csr(n, src, dst, w):
    order = np.argsort(src, kind="stable")
    adjp = np.zeros(n + 1, np.int64)
    np.add.at(adjp, np.asarray(src, np.int64) + 1, 1)
    return np.cumsum(adjp).astype(np.int32), dst[order], w[order].copy()


def _pick(which, tail_level, rng):
    top = tail_level.max()
    if which == "source_row":
        return np.flatnonzero(tail_level == top)[:1]
    if which == "upper_half":
        return rng.choice(np.flatnonzero(tail_level > top // 2), 37, replace=False)
    if which == "lowest":
        return np.flatnonzero(tail_level == tail_level.min())[:1]
    return rng.choice(tail_level.size, tail_level.size // 7, replace=False)


@pytest.mark.parametrize("heap_mode", [0, 2])
@pytest.mark.parametrize("which", ["source_row", "upper_half", "lowest", "spread"])
@pytest.mark.parametrize("name", ["small_f32_s11", "small_int_s13", "single20k_f32"])
def test_rebuild_over_known_levels_equals_oracle(name, which, heap_mode):
    n, src, dst, w = cases.load_case(name)
    adjp, adj, w = _csr(n, src, dst, w)
    tails = np.repeat(np.arange(n, dtype=np.int32), np.diff(adjp))
    rng = np.random.default_rng(7)
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, sfxt_heap_mode=heap_mode) as g:
        g.load_csr(n, adjp, adj, w)
        lvl = g.get_sfxt()[2]
        for _ in range(3):
            e = _pick(which, lvl[tails], rng).astype(np.int32)
            x = rng.integers(1, 101, e.size).astype(np.float32)
            w[e] = x
            g.update_delays(e, x)
        g.report_paths(2000)
        got = g.get_slacks(2000)
        dist, succ, lvl2 = g.get_sfxt()
    og = oracle.OracleGraph.from_edges(n, tails, adj, w)
    want = og.closure_topk(2000)[0]["slack"]
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    with cpg_b200.CpGen() as f:
        f.load_csr(n, adjp, adj, w)
        for a, b in zip((dist, succ, lvl2), f.get_sfxt()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("caller_order", [0, 1])
@pytest.mark.parametrize("graphs", [1, 3, 9])
def test_changed_side_by_side_graphs_equal_alone(graphs, caller_order):
    o, so = cpg_b200.Options(), cpg_b200.ServerOptions()
    cpg_b200.lib.cpg_options_init(C.byref(o))
    cpg_b200.lib.cpg_server_options_init(C.byref(so))
    o.batch_caller_order = caller_order
    s = cpg_b200.Server.__new__(cpg_b200.Server)
    s._s, s.ks = C.c_void_p(), {}
    assert cpg_b200.lib.cpg_server_create(C.byref(s._s), C.byref(o), C.byref(so)) == 0
    csrs = []
    for i in range(graphs):
        d = cpg_b200.generate(cpg_b200.gen_params(
            seed=70 + i, n_pins=300 + 211 * i, n_levels=5 + 3 * i, n_first=5, n_last=5, level_span=2,
            degree_kind=0, deg_lo=1, deg_hi=4))
        csrs.append([d.n, *_csr(d.n, d.src, d.dst, d.w)])
        s.add_graph(*csrs[-1])
    s.start()
    rng = np.random.default_rng(3)
    want = []
    asked = []
    for step in range(6):
        for i, c in enumerate(csrs):
            if (step + i) % 2 and graphs > 1:
                asked.append(s.submit(i, 300))
            else:
                e = rng.choice(c[2].size, 1 + 17 * step, replace=False).astype(np.int32)
                x = rng.uniform(0.1, 10.0, e.size).astype(np.float32)
                c[3][e] = x
                asked.append(s.submit(i, 300, e, x))
            with cpg_b200.CpGen() as h:
                h.load_csr(*c)
                h.report_paths(300)
                want.append(h.get_slacks(300))
    for t, x in zip(asked, want):
        assert np.array_equal(s.wait(t)[0].view(np.uint32), x.view(np.uint32))
    s.stop()
    s.close()


def test_edge_id_out_of_range_changes_nothing():
    n, src, dst, w = cases.load_case("small_f32_s11")
    adjp, adj, w = _csr(n, src, dst, w)
    with cpg_b200.CpGen() as g:
        g.load_csr(n, adjp, adj, w)
        g.report_paths(500)
        before = g.get_slacks(500)
        for bad in (-1, adj.size):
            with pytest.raises(cpg_b200.CpgError) as err:
                g.update_delays(np.array([0, 5, bad], np.int32), np.full(3, 99.0, np.float32))
            assert err.value.status == cpg_b200.CPG_ERR_INVALID
        g.levelize()
        g.report_paths(500)
        assert np.array_equal(g.get_slacks(500), before)
        assert np.array_equal(g.get_csr()[2], w)


@pytest.mark.parametrize("heap_mode", [1, 2])
@pytest.mark.parametrize("deg", [1, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 700])
def test_rows_at_the_edges_of_the_register_words(deg, heap_mode):
    """Full and known-level builds of rows of exactly `deg` edges, some with a
    parallel path of equal cost (ties), in either heap regime."""
    rng = np.random.default_rng(deg)
    width, levels = max(deg, 5), 4
    n = levels * width + 2
    src, dst = [], []
    for lv in range(levels - 1):
        for i in rng.choice(width, 9, replace=width < 9):
            heads = rng.choice(width, deg, replace=False)
            src += [lv * width + int(i)] * deg
            dst += ((lv + 1) * width + heads).tolist()
    pairs = np.unique(np.stack([src, dst], 1), axis=0)
    tails = np.setdiff1d(pairs[:, 1], pairs[:, 0])
    heads = np.setdiff1d(pairs[:, 0], pairs[:, 1])
    pairs = np.concatenate([pairs, np.stack([tails, np.full(tails.size, n - 1)], 1),
                            np.stack([np.full(heads.size, n - 2), heads], 1)])
    src, dst = pairs[:, 0].astype(np.int32), pairs[:, 1].astype(np.int32)
    w = rng.integers(1, 6, src.size).astype(np.float32)
    adjp, adj, w = _csr(n, src, dst, w)
    tail = np.repeat(np.arange(n, dtype=np.int32), np.diff(adjp))
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE, sfxt_heap_mode=heap_mode) as g:
        g.load_csr(n, adjp, adj, w)
        for step in range(2):
            og = oracle.OracleGraph.from_edges(n, tail, adj, w)
            for a, b in zip(g.get_sfxt(), og.sfxt()):
                np.testing.assert_array_equal(a, b)
            want = og.closure_topk(1500)[0]["slack"]
            g.report_paths(1500)
            assert np.array_equal(g.get_slacks(1500).view(np.uint32), want.view(np.uint32))
            e = rng.choice(adj.size, 1 + adj.size // 3, replace=False).astype(np.int32)
            w[e] = rng.integers(1, 6, e.size).astype(np.float32)
            g.update_delays(e, w[e])


@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 300])
def test_few_updates_one_by_one_equal_a_fresh_upload(count):
    n, src, dst, w = cases.load_case("small_f32_s12")
    adjp, adj, w = _csr(n, src, dst, w)
    rng = np.random.default_rng(count)
    with cpg_b200.CpGen(division=cpg_b200.DIV_IEEE) as g, cpg_b200.CpGen(division=cpg_b200.DIV_IEEE) as f:
        g.load_csr(n, adjp, adj, w)
        for step in range(3):   # before any levels, with a current tree, and twice in a row
            e = rng.choice(w.size, count, replace=False).astype(np.int32)
            w[e] = rng.uniform(0.1, 10, count).astype(np.float32)
            g.update_delays(e, w[e])
            for bad in (-1, w.size):
                with pytest.raises(cpg_b200.CpgError) as err:
                    g.update_delays(np.r_[e[:-1], bad].astype(np.int32), np.zeros(count, np.float32))
                assert err.value.status == 1
            if step != 1:
                g.report_paths(1500)
        f.load_csr(n, adjp, adj, w)
        f.report_paths(1500)
        assert np.array_equal(g.get_slacks(1500).view(np.uint32), f.get_slacks(1500).view(np.uint32))
        for a, b in zip(g.get_sfxt(), f.get_sfxt()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("graphs", [1, 127, 128, 129])
def test_few_updates_of_many_side_by_side_graphs(graphs):
    d = cpg_b200.generate(cpg_b200.gen_params(seed=5, n_pins=60, n_levels=5, n_first=3, n_last=3,
                                              level_span=2, degree_kind=0, deg_lo=1, deg_hi=3))
    adjp, adj, w = _csr(d.n, d.src, d.dst, d.w)
    e = np.arange(0, w.size, 3, dtype=np.int32)
    x = np.linspace(0.5, 9.5, e.size).astype(np.float32)
    changed = w.copy()
    changed[e] = x
    want = []
    for v in (w, changed):
        og = oracle.OracleGraph.from_edges(d.n, np.repeat(np.arange(d.n, dtype=np.int32), np.diff(adjp)), adj, v)
        want.append(og.closure_topk(30)[0]["slack"].astype(np.float32))
    with cpg_b200.Server(division=cpg_b200.DIV_IEEE) as s:
        for _ in range(graphs):
            s.add_graph(d.n, adjp, adj, w)
        s.start()
        hit = {0, graphs // 2, graphs - 1}
        for g in hit:
            got = s.wait(s.submit(g, 30, e, x))[0]
            assert np.array_equal(got.view(np.uint32), want[1].view(np.uint32)), g
        for g in range(0, graphs, 7):
            got = s.wait(s.submit(g, 30))[0]
            assert np.array_equal(got.view(np.uint32), want[g in hit].view(np.uint32)), g
