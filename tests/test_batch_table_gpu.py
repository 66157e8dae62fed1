"""The batched launch with and without its table of calls: up to 64 tiles a
block searches all calls, from 65 on the range that the table gives."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle.common import expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls", [1, 2, 63, 64, 65, 128, 129])
@pytest.mark.parametrize("vectors", [1, 65])  # of the first call's rows: one tile, or two
def test_batches_around_the_table_size(calls, vectors):
    rng = np.random.default_rng(calls)
    items, wants, outs = [], [], []
    for k in range(calls):
        P, count = 4, 4 * vectors if k == 0 else 4  # allgather tiles hold 256 vectors of all source rows
        x = rng.integers(-1000, 1001, (P, count)).astype(np.int32)
        y = torch.full((P, P * count), 77, dtype=torch.int32, device="cuda")
        items.append(("allgather", torch.from_numpy(x).cuda(), y, count, bine.INT32, P))
        wants.append(expected("allgather", x, P, count))
        outs.append(y)
    b = bine.Batch(items)
    b.launch()
    torch.cuda.synchronize()
    for k in range(calls):
        assert np.array_equal(outs[k].cpu().numpy().reshape(wants[k].shape), wants[k]), k
    b.close()


@pytest.mark.parametrize("P,count", [(456, 888), (521, 40), (97, 4), (1024, 8)])
@pytest.mark.parametrize("coll", ["allreduce", "reduce_scatter"])
def test_float_tiles_of_many_rows(coll, P, count):
    """FP64 accumulation and one rounding: within half an ulp of the FP64 sum
    and that sum's own P 2^-52 sum|x|."""
    from oracle.common import buffer_counts

    if coll == "reduce_scatter":
        count = 4
    si, so = buffer_counts(coll, count, P)
    x = np.random.default_rng(P).standard_normal((P, si)).astype(np.float32)
    y = torch.zeros((P, so), device="cuda")
    b = bine.Batch([(coll, torch.from_numpy(x).cuda(), y, count, bine.FLOAT, P)])
    b.launch()
    torch.cuda.synchronize()
    want = expected(coll, x.astype(np.float64), P, count)
    absum = expected(coll, np.abs(x).astype(np.float64), P, count)
    assert np.all(np.abs(y.cpu().numpy().reshape(want.shape) - want) <= np.abs(want) * 2.0 ** -24 + P * 2.0 ** -52 * absum)
    b.close()
