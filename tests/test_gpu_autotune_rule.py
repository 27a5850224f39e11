"""The autotuner calibrates the rules that run: the thresholds it sets follow from
the timings it returns, by the populations that each rule counts (tiles of more
than 96 bits for Four Russians, more than 4 for the tensor cores)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,densities", [((2048, 8192), (0.002, 0.02, 0.1, 0.3, 0.6)), ((1024,), (0.01, 0.3)),
                                             ((4096, 512), (0.0005, 0.4))])
def test_thresholds_follow_from_the_timings(pkg, sizes, densities):
    c = pkg.capi.Context(0)
    try:
        default = c.selector_config()
        cfg, t = c.autotune(sizes=sizes, densities=densities, reps=2)
    finally:
        c.close()
    pop = np.asarray(densities, np.float32) * 4096
    tiles = [(n + 63) // 64 for n in sizes]
    dense = pop > 96
    m4r = t[:, dense, 1].sum(dtype=np.float64) < t[:, dense, 0].sum(dtype=np.float64)
    assert cfg["m4r_min_dense"] == pytest.approx(default["m4r_min_dense"] if m4r else 1.5)
    wins = []
    for i, T in enumerate(tiles):
        count = pop > (4 if 12 <= T <= 2048 else 96)
        wins.append(t[i, count, 2].sum(dtype=np.float64) < t[i, count, :2].min(axis=1).sum(dtype=np.float64))
    assert cfg["tc_min_occ"] == pytest.approx(default["tc_min_occ"])
    if any(wins):
        smallest = min(T for T, w in zip(tiles, wins) if w)
        assert cfg["tc_min_dense"] == pytest.approx(default["tc_min_dense"])
        assert cfg["tc_min_tiles"] == (min(smallest, default["tc_min_tiles"]) if all(wins) else smallest)
    else:
        assert cfg["tc_min_dense"] == 2


def test_autotuned_selection_is_the_measured_one(pkg):
    """On this device the tensor cores are ahead at both default sizes, and Four Russians over the dense
    densities, so the defaults' rule comes out."""
    c = pkg.capi.Context(0)
    try:
        default = c.selector_config()
        cfg, _ = c.autotune(reps=10)
    finally:
        c.close()
    assert cfg == default
