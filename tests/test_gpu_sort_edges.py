"""Key-ordered output at the edges of its kernels, element by element against
the oracle: one bucket and one key more, one and two levels of splitters, key
distributions that fill the buckets' bins evenly, one by one, or all into one
(splitters inside shared memory), up to 8 aggregates (the gathered path), and more groups
than two levels of splitters take (the radix passes)."""
import numpy as np
import pytest

import cpu_oracle as O
from gpu_util import run_gpu

pytestmark = pytest.mark.gpu


def _keys(dist, n, kdt, rng):
    info = np.iinfo(kdt)
    if dist == "uniform":
        k = np.unique(rng.integers(info.min, info.max, size=2 * n + 64, endpoint=True, dtype=kdt))
    elif dist == "dense":
        k = np.arange(-(n // 2), n - n // 2)
    elif dist == "clusters":  # long gaps between short runs
        step = (int(info.max) - 64) // (n // 50 + 2)
        k = (np.arange(n // 50 + 1, dtype=object) * step)[:, None] + np.arange(50, dtype=object)[None, :]
        k = np.array(k.ravel()[:n], dtype=np.int64)
    else:  # "powers": every scale alike
        k = np.unique(np.floor(np.exp(rng.uniform(0, np.log(float(info.max)) * 0.999, size=3 * n + 64))).astype(np.int64))
    k = rng.permutation(np.asarray(k).astype(kdt))
    return k[:n]


@pytest.mark.parametrize("dist", ["uniform", "dense", "clusters", "powers"])
@pytest.mark.parametrize("n", [2, 33, 4096, 4097, 20_011, 300_007])
def test_sorted_distributions(ctx, n, dist):
    for kdt in (np.int64, np.int32):
        if dist == "powers" and kdt == np.int32 and n > 4097:
            continue  # too few distinct values
        rng = np.random.default_rng(n)
        keys = _keys(dist, n, kdt, rng)
        cols = [rng.integers(-(1 << 40), 1 << 40, size=len(keys))]
        aggs = [("sum", 0), ("count", None)]
        gk, ga, _ = run_gpu(ctx, keys, cols, aggs, knobs=dict(sort_output=1))
        ok, oa = O.groupby(keys, cols, aggs, nthreads=8)
        np.testing.assert_array_equal(gk, ok, err_msg=f"{dist} {kdt.__name__} {n}: keys")
        for g, o in zip(ga, oa):
            np.testing.assert_array_equal(g, o, err_msg=f"{dist} {kdt.__name__} {n}")


@pytest.mark.parametrize("naggs", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("n", [3000, 70_001])
def test_sorted_aggregate_counts(ctx, n, naggs):
    rng = np.random.default_rng(naggs)
    keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint32)
    cols = [rng.integers(-1000, 1000, size=n) for _ in range(4)]
    aggs = [("sum", 0), ("min", 1), ("max", 2), ("sum", 3), ("count", None), ("max", 0), ("min", 3), ("sum", 2)][:naggs]
    gk, ga, _ = run_gpu(ctx, keys, cols, aggs, knobs=dict(sort_output=1))
    ok, oa = O.groupby(keys, cols, aggs, nthreads=8)
    np.testing.assert_array_equal(gk, ok)
    for g, o in zip(ga, oa):
        np.testing.assert_array_equal(g, o)


def test_sorted_past_two_levels(ctx):
    import torch
    n = 92_000_003
    keys = (torch.arange(n, device="cuda") * 0x7FEB352D).to(torch.int32)  # distinct: an odd multiplier mod 2^32
    res = ctx.groupby(keys, [], [("count", None)], knobs=dict(sort_output=1))
    assert res.n_groups == n
    assert torch.equal(res.keys, torch.sort(keys).values)
    assert bool((res.aggs[0] == 1).all())


def test_sorted_batch_of_mixed_jobs(ctx):
    """One call whose queries take every route of the sort: empty, one bucket,
    one and two levels, both key widths, 1 to 5 aggregates."""
    from gpu_util import to_device
    rng = np.random.default_rng(4)
    aggs = [("sum", 0), ("count", None), ("max", 0), ("min", 0), ("max", 0)]
    specs = [(1, 1), (5000, 1), (4096, 2), (4097, 2), (30_000, 4), (30_000, 5), (400_003, 2), (400_003, 3), (9000, 1)]
    host, qs = [], []
    for i, (n, na) in enumerate(specs):
        kdt = (np.int64, np.int32, np.uint32)[i % 3]
        keys, cols = _keys("uniform", n, np.int64 if kdt == np.int64 else np.int32, rng).astype(kdt), \
            [rng.integers(-1000, 1000, size=n)]
        host.append((keys, cols, aggs[:na]))
        qs.append((to_device(keys), [to_device(cols[0])], aggs[:na], kdt == np.uint32))
    for (keys, cols, a), r in zip(host, ctx.groupby_batch(qs, knobs=dict(sort_output=1))):
        gk = r.keys.cpu().numpy()
        gk = gk.view(np.uint32) if keys.dtype == np.uint32 else gk
        ok, oa = O.groupby(keys, cols, a, nthreads=8)
        np.testing.assert_array_equal(gk, ok)
        for g, o in zip(r.aggs, oa):
            np.testing.assert_array_equal(g.cpu().numpy(), o)
