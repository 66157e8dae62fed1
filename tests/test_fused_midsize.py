"""Fused plans from 9 to 34 ranks: how long their programs are, how many
passes they take, and that no result is left in a workspace slot (CPU); the
plans run bit for bit like the oracle (GPU)."""
import numpy as np
import pytest

import bine_trees_fugaku_b200 as bine
from oracle import port

FUSION = 6  # levels per pass of the automatic rule for reductions


def make_comm(P, coll):
    comm = bine.Comm(P)
    if coll == "allreduce":
        comm.set_algo(coll, "B")
    comm.set_engine("pipelined")
    return comm


@pytest.mark.parametrize("P,passes,leaves", [(10, 2, 10), (16, 2, 16), (18, 3, 8), (20, 3, 8), (24, 3, 8), (30, 3, 8),
                                             (32, 3, 8), (34, 3, 16)])
def test_allreduce_plans(P, passes, leaves):
    mv, lv, dv, tmp = make_comm(P, "allreduce").plan_fused("allreduce", P * 40 + 7, 0, FUSION)
    assert len(np.unique(mv[:, 0])) == passes
    assert mv[:, 3].max() <= leaves
    assert tmp == 0 and (dv[:, 1] != 2).all()  # every pass writes receive rows only


@pytest.mark.parametrize("coll", ["reduce_scatter", "reduce"])
def test_32_ranks_take_two_passes_to_one_row_each(coll):
    mv, _, _, _ = make_comm(32, coll).plan_fused(coll, 40, 0, FUSION)
    assert len(np.unique(mv[:, 0])) == 2 and mv[:, 3].max() <= 8


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.int8])
@pytest.mark.parametrize("P,count", [(10, 1021), (18, 36), (20, 20 * 64), (24, 1697), (24, 24 * 16), (30, 4001), (32, 32 * 33), (34, 1000)])
def test_pipelined_allreduce_matches_the_oracle(P, count, dtype):
    import torch

    rng = np.random.default_rng(P + count)
    x = (rng.standard_normal((P, count)) if dtype == np.float32 else rng.integers(-128, 128, (P, count))).astype(dtype)
    want = port.run("allreduce", x, count, variant="B")[0] if dtype == np.float32 else \
        np.tile(x.sum(0, dtype=np.int8), (P, 1))
    comm = make_comm(P, "allreduce")
    comm.set_stream(torch.cuda.current_stream())
    send = torch.from_numpy(x).cuda()
    recv = torch.zeros_like(send)
    for _ in range(2):
        comm.allreduce(send, recv, count, bine.FLOAT if dtype == np.float32 else bine.CHAR)
    comm.synchronize()
    assert np.array_equal(recv.cpu().numpy().view(np.uint8), want.view(np.uint8))
    comm.close()
