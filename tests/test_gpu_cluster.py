"""Small queries in one thread-block cluster (kernel_cluster.cu) against the CPU
oracle: sizes around the rows per CTA (16, 32, 64), the tile and the cluster's
limit of 1024 vertices, sparse and dense closures (which leave for the
persistent kernel), vertex orders, epsilon rules, iteration limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(pkg, kind, n, seed):
    w = pkg.workloads
    if kind == "brackets":
        return w.Workload(kind, w.BRACKETS_GRAMMAR, w.uniform_graph(n, 3 * n, ["a", "b"], seed), {})
    if kind == "ontology":
        return w.ontology_query(n, seed)
    labels = [f"l{i}" for i in range(4)]  # grammar 5: long and sparse, 4: short and dense
    return w.Workload(kind, w.random_cnf(8, 20, labels, 5 if kind == "sparse" else 4),
                      w.uniform_graph(n, 4 * n, labels, seed), {})


def _expected(oracle, wl, tmp_path):
    gp, rp = str(tmp_path / "g.txt"), str(tmp_path / "r.txt")
    wl.write(gp, rp)
    with oracle.Problem(gp, rp) as p:
        p.closure(oracle.NAIVE, 1)
        return p.results()


def _check(ctx, wl, exp, order="auto"):
    import importlib

    pkg = importlib.import_module("cfpq-on-gpgpu_b200")
    q = pkg.query.PreparedQuery(ctx, wl.grammar, wl.graph, order=order)
    try:
        for _ in range(2):
            res = q.run()
            assert res.lines == exp
        for m in q.mats:  # populations and occupancy of the tiles written back
            bits = np.unpackbits(m.download_rows().view(np.uint8), axis=1, bitorder="little")
            occ, nnz = m.tile_stats()
            assert int(nnz.sum()) == int(bits.sum())
            occupied = np.unpackbits(occ.view(np.uint8), axis=1, bitorder="little")[:, :nnz.shape[1]]
            assert not ((nnz > 0) & (occupied == 0)).any()
        _, lines = ctx.intersection(wl.grammar.rules, q.mats, wl.graph.src, wl.graph.label, wl.graph.dst, q.off, q.lm,
                                    wl.grammar.epsilon)
        assert dict(zip(wl.grammar.nonterminals, lines)) == exp
        return res.stats
    finally:
        q.close()


@pytest.mark.parametrize("n", [2, 16, 17, 63, 64, 65, 256, 257, 512, 513, 1000, 1024, 1025])
@pytest.mark.parametrize("kind", ["brackets", "sparse", "dense"])
def test_small_queries_match_the_oracle(pkg, oracle, ctx, tmp_path, kind, n):
    wl = _workload(pkg, kind, n, n)
    _check(ctx, wl, _expected(oracle, wl, tmp_path))


@pytest.mark.parametrize("n,order", [(64, None), (300, "auto"), (900, "reverse"), (1024, "auto")])
def test_small_queries_under_a_vertex_order(pkg, oracle, ctx, tmp_path, n, order):
    wl = _workload(pkg, "ontology", n, 7)
    if order == "reverse":
        order = np.arange(wl.graph.n, dtype=np.uint32)[::-1]
    _check(ctx, wl, _expected(oracle, wl, tmp_path), order)


def test_small_query_with_epsilon_and_repeated_heads(pkg, oracle, ctx, tmp_path):
    gram = "S\nS A S\nS S S\nS S B\nT S T\nT T S\nT b\nA a\nB b\n"
    wl = pkg.workloads.Workload("eps", gram, pkg.workloads.uniform_graph(90, 150, ["a", "b"], 4), {})
    stats = _check(ctx, wl, _expected(oracle, wl, tmp_path))
    assert stats["products"] > 0 and stats["iterations"] > 1


@pytest.mark.parametrize("kind,n", [("brackets", 300), ("dense", 300), ("dense", 1024)])
def test_iteration_limit_and_rest(pkg, oracle, ctx, tmp_path, kind, n):
    """Every limit stops after that many iterations with a subset of the
    fixpoint; the closure then goes on to all of it (the dense ones leave the
    cluster within the first iterations)."""
    wl = _workload(pkg, kind, n, 3)
    exp = _expected(oracle, wl, tmp_path)
    q = pkg.query.PreparedQuery(ctx, wl.grammar, wl.graph)
    try:
        for limit in (1, 2, 4):
            q.load()
            assert ctx.closure(wl.grammar.rules, q.mats, max_iterations=limit)["iterations"] == limit
            counts = [c for _, c in ctx.hash_count_many(q.mats)]
            assert all(c <= exp[x][1] for c, x in zip(counts, wl.grammar.nonterminals))
            ctx.closure(wl.grammar.rules, q.mats)
            assert dict(zip(wl.grammar.nonterminals, ctx.hash_count_many(q.mats))) == exp
    finally:
        q.close()


def test_query_too_large_for_the_cluster(pkg, oracle, ctx, tmp_path):
    """33 nonterminals: above the cluster's 32 matrices, same answer."""
    gram = "S A B\nS A S1\nS1 S B\nA a\nB b\n" + "".join(f"X{i} S A\n" for i in range(29))
    wl = pkg.workloads.Workload("wide", gram, pkg.workloads.uniform_graph(100, 300, ["a", "b"], 2), {})
    _check(ctx, wl, _expected(oracle, wl, tmp_path))
