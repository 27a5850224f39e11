"""Statistics of a closure that runs in one thread-block cluster: what the header
promises of every closure holds for it too."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("brackets", 200), ("brackets", 300), ("ontology", 1000), ("sparse", 700)])
def test_statistics_of_a_small_query(pkg, ctx, kind, n):
    w = pkg.workloads
    if kind == "brackets":
        gram, g = w.BRACKETS_GRAMMAR, w.uniform_graph(n, 2 * n, ["a", "b"], n)
    elif kind == "ontology":
        gram, g = w.SAME_GENERATION_GRAMMAR, w.ontology_graph(n, n)
    else:
        labels = [f"l{i}" for i in range(4)]
        gram, g = w.random_cnf(8, 20, labels, 5), w.uniform_graph(n, 4 * n, labels, n)
    q = pkg.query.PreparedQuery(ctx, pkg.query.CnfGrammar.from_text(gram), g)
    try:
        q.load()
        before = sum(c for _, c in ctx.hash_count_many(q.mats))
        st = ctx.closure(q.grammar.rules, q.mats)
        new = sum(c for _, c in ctx.hash_count_many(q.mats)) - before
    finally:
        q.close()
    assert st["kernel_launches"] == 2  # prologue and cluster kernel: it stayed there
    assert st["work_items"] > 0 and st["work_items"] == sum(st["variant_items"])
    # a new word carries 1 to 64 new bits, and was merged
    assert (new + 63) // 64 <= st["new_words"] <= min(new, st["out_words"])
    words = (n + 63) // 64
    assert st["bytes_staged"] == len(q.grammar.nonterminals) * n * words * 8
    assert st["products"] >= st["iterations"] > 1
