"""The batched launch at the edges of its tiles: allgathers whose rows split
into several groups, partial vector tiles, one-rank calls, and a batch of one
call, against exact sums and copies."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle.common import buffer_counts, expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls", [
    [("allgather", 33, 4)], [("allgather", 32, 260)], [("allreduce", 1, 4)],
    [("allgather", 1, 8), ("allgather", 31, 36), ("allgather", 65, 1028), ("allgather", 200, 12), ("allreduce", 97, 1036),
     ("reduce_scatter", 40, 20), ("allreduce", 512, 4), ("reduce_scatter", 3, 4096)] * 9])
def test_batch_matches_the_collectives(calls):
    rng = np.random.default_rng(len(calls))
    items, wants, outs = [], [], []
    for k, (coll, P, count) in enumerate(calls):
        si, so = buffer_counts(coll, count, P)
        x = rng.integers(-1000, 1001, (P, si)).astype(np.float32 if k % 2 else np.int32)  # sums exact in both types
        y = torch.full((P * so + 32,), 77, dtype=torch.float32 if k % 2 else torch.int32, device="cuda")
        items.append((coll, torch.from_numpy(x).cuda(), y[16:16 + P * so], count, bine.FLOAT if k % 2 else bine.INT32, P))
        wants.append(expected(coll, x, P, count))
        outs.append(y)
    b = bine.Batch(items)
    for _ in range(2):
        b.launch()
    torch.cuda.synchronize()
    for (coll, P, count), y, want in zip(calls, outs, wants):
        got = y.cpu().numpy()
        assert np.array_equal(got[16:-16].reshape(want.shape), want), (coll, P, count)
        assert (got[:16] == 77).all() and (got[-16:] == 77).all()
    b.close()
