"""Single products in one launch (k_add_mul, k_product_tc<true>, the AUTO choice)
against the plain dense kernel: sizes around the tile, 16-tile block and plan
limits (64 * 128 and 64 * 256), empty, sparse, dense and mixed operands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, kind, rng):
    words = (n + 63) // 64
    a = np.zeros((n, words * 64), dtype=bool)
    if kind == "sparse":
        a[rng.integers(0, n, n // 2), rng.integers(0, n, n // 2)] = True
    elif kind == "dense":
        a[:, :n] = rng.random((n, n), dtype=np.float32) < 0.3
    elif kind == "mixed":  # dense rows at the top, one hub row, stray bits elsewhere
        k = max(1, n // 3)
        a[:k, :n] = rng.random((k, n), dtype=np.float32) < 0.2
        a[n - 1, :n] = True
        a[rng.integers(0, n, 40), rng.integers(0, n, 40)] = True
    return np.packbits(a, axis=1, bitorder="little").view(np.uint64)


@pytest.mark.parametrize("n", [1, 64, 65, 1000, 1025, 4097, 8192, 8193])
@pytest.mark.parametrize("kinds", [("empty", "dense"), ("sparse", "mixed"), ("dense", "sparse"), ("mixed", "dense")])
def test_add_mul_variants_agree_with_plain(ctx, n, kinds):
    rng = np.random.default_rng(n)
    a, b, c, want = (ctx.matrix(n) for _ in range(4))
    try:
        a.upload_rows(_rows(n, kinds[0], rng))
        b.upload_rows(_rows(n, kinds[1], rng))
        start = _rows(n, "sparse", rng)
        want.upload_rows(start)
        changed = ctx.add_mul(want, a, b, "plain")
        rows, stats = want.download_rows(), want.tile_stats()
        for variant in ("auto", "lop3", "m4r", "tc"):
            c.upload_rows(start)
            assert ctx.add_mul(c, a, b, variant) == changed, variant
            assert np.array_equal(c.download_rows(), rows), variant
            occ, nnz = c.tile_stats()
            assert np.array_equal(nnz, stats[1]) and np.array_equal(occ, stats[0]), variant
            assert not ctx.add_mul(c, a, b, variant), variant  # again: nothing new, the counters start over
    finally:
        for m in (a, b, c, want):
            m.destroy()


def test_add_mul_auto_at_the_plan_limit(ctx):
    """Above 64 * 256 vertices AUTO plans its product like before."""
    n = 64 * 256 + 1
    rng = np.random.default_rng(3)
    a, b, c, d = (ctx.matrix(n) for _ in range(4))
    try:
        for m in (a, b):
            m.set_bits(rng.integers(0, n, 4000), rng.integers(0, n, 4000))
        assert ctx.add_mul(c, a, b, "auto") == ctx.add_mul(d, a, b, "plain")
        assert c.hash_count() == d.hash_count()
    finally:
        for m in (a, b, c, d):
            m.destroy()
