"""The sparse loop of the word-level products: tiles whose rows hold from one to
all 64 bits (walked by lanes, or taken together by the warp), few and many such
rows, on both sides of the populations at which the dense loops take over, with
one or all Q tiles of a block occupied."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(a):
    return np.packbits(a, axis=1, bitorder="little").view(np.uint64)


@pytest.mark.parametrize("rows", [1, 2, 5, 31, 64])
@pytest.mark.parametrize("columns", [1, 16])
def test_rows_with_many_bits(ctx, rows, columns):
    n, rng = 1280, np.random.default_rng(rows)
    for bits in (1, 4, 5, 8, 9, 13, 40, 64):
        a, b = np.zeros((n, n), dtype=bool), np.zeros((n, n), dtype=bool)
        for ti, tk in ((0, 0), (3, 7), (19, 19), (19, 2)):
            for r in rng.choice(64, rows, replace=False):
                a[64 * ti + r, 64 * tk + rng.choice(64, bits, replace=False)] = True
        b[:, :64 * columns] = rng.random((n, 64 * columns), dtype=np.float32) < 0.05
        want = (a.astype(np.float32) @ b.astype(np.float32)) > 0  # counts below 2^24: exact
        ma, mb, mc = (ctx.matrix(n) for _ in range(3))
        try:
            ma.upload_rows(_pack(a))
            mb.upload_rows(_pack(b))
            for variant in ("lop3", "m4r"):
                mc.clear()
                ctx.add_mul(mc, ma, mb, variant)
                assert np.array_equal(mc.download_rows(), _pack(want)), (bits, variant)
            mc.clear()  # the persistent kernel's split of the tiles over warps
            ctx.closure([(2, 0, 1)], [ma, mb, mc], driver="engine", variant="lop3")
            assert np.array_equal(mc.download_rows(), _pack(want)), bits
        finally:
            for m in (ma, mb, mc):
                m.destroy()
