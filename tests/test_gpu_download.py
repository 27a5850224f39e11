"""Rows on their way to the host: sizes on both sides of a pinned chunk (1 MiB)
and of the rows that a gathering block takes (8, 4, 2, 1), in vertex order and in
another one, to pageable and to pinned memory."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 65, 333, 2880, 2944, 5003, 24577, 24700, 49200, 98400])
@pytest.mark.parametrize("ordered", [False, True])
def test_download_rows(ctx, n, ordered):
    rng = np.random.default_rng(n)
    order = ctx.order(rng.permutation(n).astype(np.uint32)) if ordered else None
    m = ctx.matrix(n, order)
    try:
        k = min(4 * n, 50000)
        r, c = (rng.integers(0, n, k, dtype=np.int64) for _ in range(2))
        r[:3], c[:3] = (0, n - 1, n - 1), (n - 1, 0, n - 1)
        m.set_bits(r.astype(np.uint32), c.astype(np.uint32))
        got = m.download_rows()
        want = np.zeros_like(got)
        np.bitwise_or.at(want, (r, c // 64), np.uint64(1) << (c % 64).astype(np.uint64))
        assert np.array_equal(got, want)
        if n <= 5003:
            pinned = torch.zeros(got.shape, dtype=torch.int64, pin_memory=True)
            assert ctx.lib.cfpq_matrix_download_rows(ctx.handle, m.handle, ctypes.c_void_p(pinned.data_ptr())) == 0
            assert np.array_equal(pinned.numpy().view(np.uint64), want)
    finally:
        m.destroy()
        if order is not None:
            order.destroy()
