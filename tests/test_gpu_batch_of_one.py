"""cfpq_closure_batch with a single query: a dense one starts in the cluster's or
the persistent kernel and goes on in others, and its per-query results are those
of the whole closure, not of the stage that it began in."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loop", ["device", "graph", "host"])
@pytest.mark.parametrize("kind,n", [("dense", 300), ("dense", 1089), ("dense", 2000), ("brackets", 1024),
                                    ("brackets", 200)])
def test_iterations_and_time_of_a_single_query(pkg, ctx, kind, n, loop):
    w = pkg.workloads
    if kind == "dense":
        labels = [f"l{i}" for i in range(4)]
        gram, g = w.random_cnf(8, 20, labels, 4), w.uniform_graph(n, 4 * n, labels, n)
    else:
        gram, g = w.BRACKETS_GRAMMAR, w.uniform_graph(n, 4 * n, ["a", "b"], n)
    q = pkg.query.PreparedQuery(ctx, pkg.query.CnfGrammar.from_text(gram), g)
    try:
        for _ in range(2):
            q.load()
            t0 = time.perf_counter()
            st, iters, done = ctx.closure_batch([(q.grammar.rules, q.mats)], use_graph=loop)
            wall = (time.perf_counter() - t0) * 1e3
            if loop != "host":  # (host iterations come in fours, the surplus ones do nothing)
                # the last iteration finds nothing new
                assert int(iters[0]) == st["iterations"] - 1
            if loop == "device" and kind == "dense":
                assert st["kernel_launches"] > 2  # more than prologue and closure: it changed kernels
            assert 0 < done[0] <= wall
    finally:
        q.close()
