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
