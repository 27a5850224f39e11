"""Selection on both sides of the sizes at which the dense-tile limit changes
(12 tiles) and of the single product's tensor-core size (32 tiles): closures and
products by AUTO equal those of the plain driver and kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [704, 705, 1024])
def test_closure_around_the_dense_limit(pkg, ctx, n):
    labels = [f"l{i}" for i in range(4)]
    g = pkg.workloads.uniform_graph(n, 4 * n, labels, n)
    gram = pkg.query.CnfGrammar.from_text(pkg.workloads.random_cnf(8, 20, labels, 4))
    answers = [pkg.query.run_query(ctx, gram, g, driver="engine", variant=v).lines for v in ("auto", "lop3")]
    assert answers[0] == answers[1]


@pytest.mark.parametrize("n", [2047, 1984, 2049])
@pytest.mark.parametrize("bits", [0.002, 0.003, 0.006])
def test_single_product_around_the_limits(ctx, n, bits):
    rng = np.random.default_rng(n)
    words = (n + 63) // 64
    rows = np.zeros((n, words * 64), dtype=bool)
    rows[:, :n] = rng.random((n, n), dtype=np.float32) < bits
    packed = np.packbits(rows, axis=1, bitorder="little").view(np.uint64)
    a, c, want = (ctx.matrix(n) for _ in range(3))
    try:
        a.upload_rows(packed)
        assert ctx.add_mul(want, a, a, "plain") == ctx.add_mul(c, a, a, "auto")
        assert np.array_equal(c.download_rows(), want.download_rows())
        assert ctx.add_mul(c, a, a, "auto") is False
    finally:
        for m in (a, c, want):
            m.destroy()
