"""Which tiles the selector counts for which rule: Four Russians and the cost
model's features go by tiles of more than 96 bits, the tensor cores by tiles of
more than 4 (12 to 2048 tile rows) -- whether or not the tensor cores may run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOG_SELECTION = 4
N = 1089  # 18 tile rows


def _tiles(rng, n, bits, share):
    """Row bits with `bits` bits in every whole tile of a random share of the tiles (the
    ragged last tile row and column stay empty)."""
    full = n // 64
    m = np.zeros((n, (n + 63) // 64 * 64), dtype=bool)
    for i in range(full):
        for j in range(full):
            if rng.random() < share:
                k = rng.permutation(4096)[:bits]
                m[64 * i + k // 64, 64 * j + k % 64] = True
    return np.packbits(m, axis=1, bitorder="little").view(np.uint64)


def _first_iteration(ctx, allowed, bits, share=1.0):
    """(variant items, features of the first product) of a batch of two C -> A B."""
    before = ctx.selector_config()
    ctx.selector_configure(allowed=allowed, mode="heuristic")
    rng = np.random.default_rng(bits)
    mats = [[ctx.matrix(N) for _ in range(3)] for _ in range(2)]
    try:
        for _, a, b in mats:
            a.upload_rows(_tiles(rng, N, bits, share))
            b.upload_rows(_tiles(rng, N, bits, share))
        st, _, _ = ctx.closure_batch([([(0, 1, 2)], m) for m in mats], max_iterations=1, log_products=LOG_SELECTION)
        return st["variant_items"], np.asarray(ctx.product_log()[0]["features"])
    finally:
        for m in sum(mats, []):
            m.destroy()
        ctx.selector_configure(**before)


def _used(items):
    names = ("auto", "plain", "lop3", "m4r", "tc")
    values = items.values() if isinstance(items, dict) else items
    return {n for n, v in zip(names, values) if v}


@pytest.mark.parametrize("bits,used", [(5, {"lop3"}), (20, {"lop3"}), (96, {"lop3"}), (97, {"m4r"}), (300, {"m4r"})])
def test_four_russians_limit_without_tensor_cores(ctx, bits, used):
    items, f = _first_iteration(ctx, ["lop3", "m4r"], bits)
    assert _used(items) == used
    assert f[6] == f[7] == (bits > 96)


@pytest.mark.parametrize("bits,used", [(4, {"lop3"}), (5, {"tc"}), (96, {"tc"}), (300, {"tc"})])
def test_tensor_core_limit(ctx, bits, used):
    items, f = _first_iteration(ctx, ["lop3", "m4r", "tc"], bits)
    assert _used(items) == used
    assert f[6] == f[7] == (bits > 96)


@pytest.mark.parametrize("bits,used", [(20, {"lop3"}), (300, {"m4r"})])
def test_few_occupied_tiles_fall_back_by_their_own_limit(ctx, bits, used):
    """Below the tensor cores' occupied share, light tiles are no case for Four Russians."""
    items, _ = _first_iteration(ctx, ["lop3", "m4r", "tc"], bits, share=0.05)
    assert _used(items) == used


@pytest.mark.parametrize("n,tensor", [(704, False), (705, True)])
def test_closure_on_both_sides_of_the_tensor_core_size(pkg, oracle, ctx, tmp_path, n, tensor):
    """Selection forced from the start (min_tiles 1), against the CPU oracle."""
    w = pkg.workloads
    labels = [f"l{i}" for i in range(4)]
    wl = w.Workload("dense", w.random_cnf(8, 20, labels, 4), w.uniform_graph(n, 4 * n, labels, n), {})
    gp, rp = str(tmp_path / "g.txt"), str(tmp_path / "r.txt")
    wl.write(gp, rp)
    with oracle.Problem(gp, rp) as p:
        p.closure(oracle.NAIVE, 1)
        exp = p.results()
    before = ctx.selector_config()
    ctx.selector_configure(min_tiles=1)
    try:
        res = pkg.query.run_query(ctx, wl.grammar, wl.graph)
    finally:
        ctx.selector_configure(**before)
    assert res.lines == exp
    assert ("tc" in _used(res.stats["variant_items"])) == tensor
