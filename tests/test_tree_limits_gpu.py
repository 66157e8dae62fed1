"""Exact-order float reductions whose programs leave no room in shared memory
for the split form, reached with small calls through a lowered limit."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [2, 4, 8])
@pytest.mark.parametrize("P,count", [(96, 4097), (64, 65)])
def test_rows_off_the_grid_without_room_for_the_split(P, count, lanes):
    x = np.random.default_rng(P + lanes).standard_normal((P, count)).astype(np.float32)
    send = torch.from_numpy(x).cuda()
    comm = bine.Comm(P)
    comm.set_stream(torch.cuda.current_stream())
    comm.set_tree_split(lanes)
    expect, _ = port.run("allreduce", x, count, variant="B")
    # A program of P entries of 16 bytes fits, with the parts' 8 KB of partial
    # sums it does not.
    comm.debug_set_tree_smem_limit(4096)
    with pytest.raises(bine.BineError):
        comm.debug_set_tree_smem_limit(1 << 20)
    before = bine.last_error()
    recv = torch.zeros_like(send)
    comm.allreduce(send, recv, count, bine.FLOAT)
    comm.synchronize()
    assert np.array_equal(recv.cpu().numpy().view(np.uint32), expect.view(np.uint32))
    assert bine.last_error() == before  # the call did not fail on the way
    comm.debug_set_tree_smem_limit(16 * P - 16)
    with pytest.raises(bine.Unsupported):
        comm.allreduce(send, recv, count, bine.FLOAT)
    comm.close()
