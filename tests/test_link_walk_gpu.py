"""The two device paths of bine_link_bytes for generated schedules: the walk
of every rank's subtree (rings above the limit) on tori small enough for the
host restatement, and rings of several nodes per thread with uneven blocks."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine

pytestmark = pytest.mark.gpu


def link_bytes(dims, coll, variant, ports, family, count, limit=None):
    comm = bine.Comm(int(np.prod(dims)), dims)
    comm.set_ports(ports)
    comm.set_algo(coll, variant, family)
    comm.set_stream(torch.cuda.current_stream())
    if limit is not None:
        comm.debug_set_link_ring_limit(limit)
    out = torch.full((comm.nranks * len(dims) * 2,), -1, dtype=torch.int64, device="cuda")
    comm.link_bytes(coll, count, bine.INT32, out)
    comm.synchronize()
    host = comm.link_bytes_host(coll, count, bine.INT32)
    comm.close()
    return out.cpu().numpy().view(np.uint64), host


@pytest.mark.parametrize("dims,coll,variant,ports,family,count", [
    ([64], "allreduce", "B", 1, "BINE", 64 * 3 + 29), ([8, 16], "allreduce", "B", 4, "BINE", 4 * 128 * 3 + 77),
    ([2, 8, 4], "allreduce", "B", 6, "BINE", 6 * 64 * 2 + 5), ([16, 4], "allreduce", "B", 1, "RECDOUB", 64 * 3 + 11),
    ([32, 2], "allreduce", "L", 2, "BINE", 1001), ([16, 8], "allgather", "VEC_DOUBLING_CONT_PERMUTE", 1, "BINE", 33)])
def test_the_walk_matches_the_host(dims, coll, variant, ports, family, count):
    got, host = link_bytes(dims, coll, variant, ports, family, count, limit=max(dims) - 1)
    assert np.array_equal(got, host)


def test_a_ring_above_the_default_limit():
    got, host = link_bytes([16384], "allreduce", "L", 1, "BINE", 1001)
    assert np.array_equal(got, host)


def test_uneven_blocks_on_a_ring_of_two_nodes_per_thread():
    got, host = link_bytes([2048], "allreduce", "B", 1, "BINE", 2048 * 3 + 1365)
    assert np.array_equal(got, host)
