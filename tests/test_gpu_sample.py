"""Plain sizing of more than 2^20 rows, whose route a row sample decides:
few groups (table), many (partition by the sampled estimate), samples that
mislead (a period of the rows, a rare half of the keys, a skewed tail, sorted
keys), against the oracle."""
import numpy as np
import pytest

from gpu_util import compare, run_gpu

pytestmark = pytest.mark.gpu

AGGS = [("sum", 0), ("count", None), ("min", 0)]
N = (1 << 20) + 4099


def _keys(kind, n, rng):
    i = np.arange(n)
    return {"few": lambda: rng.integers(0, 37, n),
            "table_edge": lambda: rng.integers(0, 3000, n),
            "mid": lambda: rng.integers(0, 60_000, n),
            "distinct": lambda: rng.permutation(n),
            "periodic": lambda: i % 4096,
            "rare_half": lambda: np.where(rng.random(n) < 0.6, rng.integers(0, 20, n), 1000 + rng.permutation(n)),
            "hidden": lambda: np.where(rng.random(n) < 0.9999, 7, 1000 + i),  # most samples see one key
            "skewed": lambda: np.minimum(rng.zipf(1.3, n), 1 << 40),
            "sorted": lambda: np.sort(rng.integers(0, 200_000, n)),
            "all_ones": lambda: np.full(n, -1)}[kind]()


@pytest.mark.parametrize("kind", ["few", "table_edge", "mid", "distinct", "periodic", "rare_half", "hidden", "skewed",
                                  "sorted", "all_ones"])
@pytest.mark.parametrize("kdt", [np.int64, np.uint32])
def test_plain_sampled_routes(ctx, kind, kdt):
    rng = np.random.default_rng(11)
    keys = _keys(kind, N, rng).astype(kdt)
    cols = [rng.integers(-(1 << 40), 1 << 40, size=N)]
    gk, ga, res = run_gpu(ctx, keys, cols, AGGS)
    if kind in ("few", "all_ones"):
        assert res.stats["strategy"] == 1
    if kind in ("mid", "distinct", "rare_half"):
        assert res.stats["strategy"] == 2
    compare(gk, ga, keys, cols, AGGS, f"{kind} {np.dtype(kdt).name}")


def test_plain_sampled_table_overflow(ctx):
    """Groups that the sample cannot see overflow its table; the rows are then
    partitioned by their count."""
    n = 1 << 22
    rng = np.random.default_rng(5)
    i = np.arange(n)
    keys = np.where(i % 512 < 500, 3, 10 + i)  # 98% one key ...
    lo = n * np.arange(8192) // 8192
    hi = n * (np.arange(8192) + 1) // 8192
    jitter = ((np.arange(1, 8193, dtype=object) * 0x9e3779b97f4a7c15) % (1 << 64)) * (hi - lo) >> 64
    keys[(lo + jitter.astype(np.int64))] = 3   # ... and every sampled row holds it
    cols = [rng.integers(0, 100, size=n)]
    gk, ga, res = run_gpu(ctx, keys, cols, AGGS)
    assert res.stats["strategy"] == 2 and res.stats["regrows"] >= 1
    compare(gk, ga, keys, cols, AGGS, "hidden from the sample")
