"""Tensor-core products whose k-lists end inside an operand stage (8 k-tiles), a
unit of loads (4) or an item's half: P occupies `kcount` chosen tile columns, Q
only some tile columns of each block of four, so that halves are missing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(a):
    n = a.shape[0]
    full = np.zeros((n, (n + 63) // 64 * 64), dtype=bool)
    full[:, :n] = a
    return np.packbits(full, axis=1, bitorder="little").view(np.uint64)


@pytest.mark.parametrize("tiles", [5, 18, 33])
@pytest.mark.parametrize("columns", [(0,), (2, 3), (1, 2)])
def test_tc_partial_stages(ctx, tiles, columns):
    n = 64 * tiles - 7
    rng = np.random.default_rng(tiles * 10 + columns[0])
    for kcount in (1, 3, 4, 5, 8, 9, 16, 17, 33):
        if kcount > tiles:
            break
        ks = rng.choice(tiles, kcount, replace=False)
        used = np.isin(np.arange(n) // 64, ks)
        a = (rng.random((n, n), dtype=np.float32) < 0.02) & used[None, :]
        b = (rng.random((n, n), dtype=np.float32) < 0.02) & np.isin((np.arange(n) // 64) % 4, columns)[None, :]
        want = (a.astype(np.float32) @ b.astype(np.float32)) > 0  # counts below 2^24: exact
        ma, mb, mc = (ctx.matrix(n) for _ in range(3))
        try:
            ma.upload_rows(_pack(a))
            mb.upload_rows(_pack(b))
            assert ctx.add_mul(mc, ma, mb, "tc") == bool(want.any())
            assert np.array_equal(mc.download_rows(), _pack(want)), kcount
        finally:
            for m in (ma, mb, mc):
                m.destroy()


@pytest.mark.parametrize("seed", range(4))
def test_tc_rows_of_short_halves(ctx, seed):
    """Many items a CTA whose halves take one, two or no stages in any order: a
    group of expanders that has no stage in a row of halves must not run ahead."""
    tiles, rng = 150, np.random.default_rng(seed)
    n = 64 * tiles
    occupied = rng.random((tiles, tiles), dtype=np.float32) < rng.choice([0.005, 0.02, 0.06], tiles)[:, None]
    a = np.zeros((n, n), dtype=bool)
    for ti, tk in zip(*np.nonzero(occupied)):
        a[64 * ti + rng.integers(0, 64, 8), 64 * tk + rng.integers(0, 64, 8)] = True
    b = (rng.random((n, n), dtype=np.float32) < 0.01) & np.repeat(np.repeat(
        rng.random((tiles, tiles), dtype=np.float32) < 0.5, 64, axis=0), 64, axis=1)
    ma, mb, mc, want = (ctx.matrix(n) for _ in range(4))
    try:
        ma.upload_rows(_pack(a))
        mb.upload_rows(_pack(b))
        ctx.add_mul(want, ma, mb, "lop3")
        rows = want.download_rows()
        for _ in range(10):
            mc.clear()
            ctx.add_mul(mc, ma, mb, "tc")
            assert np.array_equal(mc.download_rows(), rows)
    finally:
        for m in (ma, mb, mc, want):
            m.destroy()
