"""Tables that travel in a kernel's arguments (short ones) or through device
buffers (long ones), and edges read in place, from the pinned stage or copied:
queries on both sides of every limit take turns on one context, and each gives
the oracle's lines every time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wide(nonterminals):
    return "S A B\nS A S1\nS1 S B\nA a\nB b\n" + "".join(f"X{i} S A\n" for i in range(nonterminals - 4))


def _expected(oracle, wl, tmp_path):
    gp, rp = str(tmp_path / "g.txt"), str(tmp_path / "r.txt")
    wl.write(gp, rp)
    with oracle.Problem(gp, rp) as p:
        p.closure(oracle.NAIVE, 1)
        return p.results()


def test_queries_around_the_table_limits_take_turns(pkg, oracle, ctx, tmp_path):
    w = pkg.workloads
    # nonterminals: 4, 36 / 37 (clear list), 42 / 43 (scatter tables), 100 (closure tables);
    # edges: 600, 21845 (the pinned stage exactly), 21846 (copied)
    cases = [(4, 70, 600), (36, 70, 150), (37, 70, 150), (42, 65, 150), (43, 65, 150), (100, 64, 100),
             (4, 500, 21845), (4, 500, 21846), (43, 65, 21846)]
    wls = [w.Workload("t", _wide(nt), w.uniform_graph(n, e, ["a", "b"], nt + e), {}) for nt, n, e in cases]
    exp = [_expected(oracle, x, tmp_path) for x in wls]
    qs = [pkg.query.PreparedQuery(ctx, x.grammar, x.graph) for x in wls]
    try:
        rng = np.random.default_rng(1)
        for i in list(range(len(qs))) * 2 + rng.integers(0, len(qs), 30).tolist():
            q, g = qs[i], wls[i].graph
            if rng.random() < 0.5:
                assert q.run().lines == exp[i], cases[i]
            else:
                _, lines = ctx.intersection(q.grammar.rules, q.mats, g.src, g.label, g.dst, q.off, q.lm)
                assert dict(zip(q.grammar.nonterminals, lines)) == exp[i], cases[i]
    finally:
        for q in qs:
            q.close()


@pytest.mark.parametrize("edges", [100, 21846])
def test_out_of_range_edges_are_counted_once_per_load(pkg, ctx, edges):
    w = pkg.workloads
    g = w.uniform_graph(200, edges, ["a", "b"], 3)
    q = pkg.query.PreparedQuery(ctx, pkg.query.CnfGrammar.from_text(w.BRACKETS_GRAMMAR), g, order=None)
    try:
        bad = g.dst.copy()
        bad[:7] = 200  # one past the last vertex
        for _ in range(2):
            with pytest.raises(pkg.capi.CfpqError, match="7 coordinates out of range"):
                ctx.load_edges(q.mats, g.src, g.label, bad, q.off, q.lm)
            ctx.load_edges(q.mats, g.src, g.label, g.dst, q.off, q.lm)  # the count starts over
    finally:
        q.close()
