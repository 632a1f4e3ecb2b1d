"""The partition kernels at their edges, against the oracle: tiles that start
off a 16-byte boundary, tile and granule remainders, every column count and
width mix, both scatter shapes, one and two passes, more partitions than one
sweep counts, a table filled beyond its buckets' homes."""
import numpy as np
import pytest

from gpu_util import compare, to_device
from test_gpu_parity import _data

pytestmark = pytest.mark.gpu

SUMS = {0: [("count", None)],
        1: [("sum", 0), ("count", None)],
        2: [("sum", 0), ("count", None), ("sum", 1)],
        3: [("sum", 0), ("min", 2), ("sum", 1), ("count", None)],
        4: [("sum", 0), ("sum", 1), ("sum", 2), ("max", 3), ("count", None)]}


def _run(ctx, n, kdt, ndv, ncols, offset, knobs, seed, zipf=0.0):
    import torch
    keys, cols = _data(n, kdt, ndv, seed=seed, zipf=zipf)
    cols = cols[:ncols]

    def dev(a):  # a slice that starts `offset` elements into its allocation
        t = to_device(a)
        room = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)
        room[offset:] = t
        return room[offset:]

    res = ctx.groupby(dev(keys), [dev(c) for c in cols], SUMS[ncols], knobs=dict(strategy="partition", **knobs),
                      unsigned_keys=kdt == np.uint32, unsigned_cols=[c.dtype == np.uint32 for c in cols])
    gk = res.keys.cpu().numpy()
    gk = gk.view(np.uint32) if kdt == np.uint32 else gk
    compare(gk, [a.cpu().numpy() for a in res.aggs], keys, cols, SUMS[ncols], f"n={n} cols={ncols} {knobs}")
    return res


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("n,bits", [(1, 1), (3, 9), (511, 2), (4095, 1), (4097, 10), (70_001, 9), (70_001, 16)])
def test_partition_tile_edges(ctx, n, bits, offset):
    for ncols in range(5):
        kdt = (np.int64, np.int32, np.uint32)[(n + ncols) % 3]
        _run(ctx, n, kdt, max(1, n // 3), ncols, offset, dict(partition_bits=bits), seed=n + ncols)


@pytest.mark.parametrize("kdt", [np.int32, np.int64])
@pytest.mark.parametrize("ndv,bits", [(700, 1), (2600, 1), (300_000, 7)])
def test_partition_table_fill(ctx, kdt, ndv, bits):
    # up to nearly as many groups in a partition as its table has slots: rows
    # walk on from full home buckets, and those without a slot use the HBM table
    _run(ctx, 600_007, kdt, ndv, 1, 1, dict(partition_bits=bits), seed=ndv)
    _run(ctx, 600_007, kdt, ndv, 4, 0, dict(partition_bits=bits, smem_slots=512), seed=ndv + 1, zipf=1.1)
