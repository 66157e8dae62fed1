"""Fused passes whose programs have up to 16 leaves: how the planner cuts a
schedule into passes (CPU), and the kernel's two forms (sums and copies),
full and uneven trees, vectors and elements off the 16-byte grid (GPU, bit
for bit against the oracle in the reference's float order)."""
import numpy as np
import pytest

import bine_trees_fugaku_b200 as bine
from oracle import port
from oracle.common import buffer_counts, expected, receiving_ranks

CODE = {np.dtype(np.int32): bine.INT32, np.dtype(np.int64): bine.INT64, np.dtype(np.float32): bine.FLOAT,
        np.dtype(np.float64): bine.DOUBLE, np.dtype(np.int8): bine.CHAR}


def make_comm(P, coll, variant, levels=0):
    comm = bine.Comm(P)
    if variant:
        comm.set_algo(coll, variant)
    comm.set_engine("pipelined")
    comm.set_fusion(levels)
    return comm


@pytest.mark.parametrize("P,count,passes,bound", [(64, 4096, 3, 1.13), (96, 9600, 3, 1.13), (128, 4096, 3, 1.13),
                                                  (256, 4096, 3, 1.13), (200, 2000, 3, 1.15)])
def test_passes_end_where_the_programs_outgrow_the_kernel(P, count, passes, bound):
    comm = make_comm(P, "allreduce", "B")
    mv, lv, _, _ = comm.plan_fused("allreduce", count, 0, 6)
    assert len(np.unique(mv[:, 0])) == passes
    assert mv[:, 3].max() == 16 and mv[:, 5].max() <= 8
    assert (mv[:, 1] * (mv[:, 3] + mv[:, 5])).sum() <= bound * 2 * P * count


@pytest.mark.parametrize("P", [2, 4, 6, 8])
def test_up_to_eight_ranks_run_in_one_pass(P):
    comm = make_comm(P, "allreduce", "B")
    _, items, _ = comm.plan_flow("allreduce", 64 * P, 0, 4, 444)
    assert items[:, 4].max() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32])
@pytest.mark.parametrize("coll,variant,P,count,levels,off", [
    ("allreduce", "B", 4, 64, 0, 0), ("allreduce", "B", 8, 1001, 0, 0), ("allreduce", "B", 8, 8 * 512, 0, 1),
    ("allreduce", "B", 16, 16, 0, 0), ("allreduce", "B", 32, 32 * 33, 0, 0), ("allreduce", "B", 76, 76 * 40 + 3, 0, 0),
    ("allreduce", "B", 96, 96 * 64, 0, 0), ("allreduce", "B", 200, 200 * 12, 0, 1), ("allreduce", "B", 256, 256, 0, 0),
    ("allreduce", "B", 256, 256 * 68, 0, 0), ("allreduce", "L", 32, 517, 0, 0), ("allreduce", "L", 16, 128, 64, 0),
    ("reduce_scatter", None, 64, 65, 0, 0), ("reduce_scatter", None, 128, 64, 0, 0), ("reduce", None, 64, 999, 0, 0),
    ("allgather", None, 64, 33, 0, 0), ("alltoall", None, 64, 36, 0, 1), ("bcast", None, 128, 1001, 0, 0)])
def test_pipelined_programs_match_the_oracle(coll, variant, P, count, levels, off, dtype):
    import torch

    si, so = buffer_counts(coll, count, P)
    rng = np.random.default_rng(P + count)
    whole = dtype == np.int32 or (dtype == np.float64 and coll not in ("allreduce",))
    x = (rng.integers(-1000, 1001, (P, si)) if whole else rng.standard_normal((P, si))).astype(dtype)
    if coll == "bcast":
        want = np.tile(x[:1], (P, 1))
    elif whole or coll in ("allgather", "alltoall"):
        want = expected(coll, x, P, count)
    else:
        want, _ = port.run(coll, x, count, **({"variant": variant} if variant else {}))
    comm = make_comm(P, coll, variant, levels)
    comm.set_stream(torch.cuda.current_stream())
    td = torch.from_numpy(x[:1, :1]).dtype
    send = torch.zeros(P * si + off, dtype=td, device="cuda")[off:].view(P, si)
    send.copy_(torch.from_numpy(x))
    pool = torch.full((P * so + off + 16,), 77, dtype=td, device="cuda")
    recv = pool[off:off + P * so].view(P, so)
    if coll == "bcast":
        recv[0] = send[0]
    rr = receiving_ranks(coll, P, 0)
    for _ in range(2):
        comm.run(coll, send, recv, count, CODE[x.dtype], 0)
        comm.synchronize()
        got = recv.cpu().numpy()
        assert np.array_equal(got[rr].view(np.uint8), want[rr].view(np.uint8))
        assert (pool[off + P * so:] == 77).all() and (pool[:off] == 77).all()
    comm.close()
