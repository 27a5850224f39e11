"""Dense closures: rules whose two semi-naive terms are merged into one product
of the current matrices (select_device.cuh merge_terms), and single queries
that leave the persistent kernel for the selecting multi-kernel loop once their
iterations are heavy.  Every result against the CPU oracle; sizes around tile,
16-tile block and 4 x 4-tile tensor-core block edges."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def sctx(pkg):
    c = pkg.capi.Context(0)
    yield c
    c.close()


def _dense(pkg, n, seed):
    """A random CNF query whose closure is dense (most of every matrix set)."""
    labels = [f"l{i}" for i in range(4)]
    return pkg.workloads.Workload("dense", pkg.workloads.random_cnf(8, 20, labels, 4),
                                  pkg.workloads.uniform_graph(n, 4 * n, labels, seed), {})


def _expected(oracle, wl, tmp_path):
    gp, rp = str(tmp_path / "g.txt"), str(tmp_path / "r.txt")
    wl.write(gp, rp)
    with oracle.Problem(gp, rp) as p:
        p.closure(oracle.M4RM, 0)
        return p.results()


@pytest.mark.parametrize("n", [1023, 1089, 2049])
def test_heavy_single_query_goes_on_with_selection(pkg, oracle, sctx, tmp_path, n):
    wl = _dense(pkg, n, n)
    exp = _expected(oracle, wl, tmp_path)
    q = pkg.query.PreparedQuery(sctx, wl.grammar, wl.graph)
    small = pkg.workloads.brackets_query(200, 800, 3)
    sexp = _expected(oracle, small, tmp_path)
    sq = pkg.query.PreparedQuery(sctx, small.grammar, small.graph)
    try:
        for _ in range(2):  # again on the same plan and buffers, another query in between
            res = q.run()
            assert res.lines == exp
            items = res.stats["variant_items"]
            assert items[pkg.capi.VARIANT_TC] + items[pkg.capi.VARIANT_M4R] > 0  # it left the LOP3-only kernel
            assert sq.run().lines == sexp
        st, lines = sctx.intersection(wl.grammar.rules, q.mats, wl.graph.src, wl.graph.label, wl.graph.dst, q.off, q.lm)
        assert dict(zip(wl.grammar.nonterminals, lines)) == exp
        # an iteration limit after the kernel has left, then the rest
        q.load()
        assert sctx.closure(wl.grammar.rules, q.mats, max_iterations=3)["iterations"] == 3
        sctx.closure(wl.grammar.rules, q.mats)
        assert dict(zip(wl.grammar.nonterminals, sctx.hash_count_many(q.mats))) == exp
    finally:
        q.close()
        sq.close()


@pytest.mark.parametrize("n", [577, 1025])
@pytest.mark.parametrize("loop,allowed", [("graph", ["lop3", "m4r", "tc"]), ("host", ["lop3", "m4r", "tc"]),
                                          ("graph", ["lop3"]), ("device", ["lop3", "m4r"])])
def test_merged_rules_in_every_loop(pkg, oracle, sctx, tmp_path, n, loop, allowed):
    """A batch (selection from the first iteration): merged rules on the
    tensor cores, in the word-level kernels and in the persistent kernel."""
    sctx.selector_configure(mode="heuristic", min_tiles=1, tc_min_tiles=1, allowed=allowed)
    wls = [_dense(pkg, n, 1), _dense(pkg, 130, 2), pkg.workloads.chain_query(700, 5)]
    exp = [_expected(oracle, w, tmp_path) for w in wls]
    qs = [pkg.query.PreparedQuery(sctx, w.grammar, w.graph) for w in wls]
    try:
        for q in qs:
            q.load()
        sctx.closure_batch([(q.grammar.rules, q.mats) for q in qs], use_graph=loop)
        for q, e in zip(qs, exp):
            assert dict(zip(q.grammar.nonterminals, sctx.hash_count_many(q.mats))) == e
    finally:
        for q in qs:
            q.close()
