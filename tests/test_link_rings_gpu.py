"""bine_link_bytes ring by ring (k_link_rings) against the host restatement
(bine_link_bytes_host), exactly: rings from 2 nodes to several per thread,
uneven blocks in every position of the torus order, single- and multi-port."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine

pytestmark = pytest.mark.gpu


def check(dims, coll, variant, ports, family, count):
    P = int(np.prod(dims))
    comm = bine.Comm(P, dims)
    comm.set_ports(ports)
    comm.set_algo(coll, variant, family)
    comm.set_stream(torch.cuda.current_stream())
    host = comm.link_bytes_host(coll, count, bine.INT32)
    out = torch.full((len(host),), -1, dtype=torch.int64, device="cuda")  # every link is written
    comm.link_bytes(coll, count, bine.INT32, out)
    comm.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), host), (dims, coll, variant, ports, family, count)
    comm.close()


@pytest.mark.parametrize("dims", [[2], [64], [512], [2, 64], [64, 4], [8, 16], [2, 2, 2], [32, 4, 2], [2, 16, 8],
                                  [8, 2, 16]])
@pytest.mark.parametrize("ports", [1, 2, 6])
def test_uneven_blocks_match_the_host(dims, ports):
    """Allreduce B: the first `rem` ranks' blocks hold one element more; rem
    from 0 to P - 1 cuts the ranks anywhere in the lexicographic order."""
    P = int(np.prod(dims))
    for extra in sorted({0, 1, P // 2, P // 2 + 1, P - 1, (5 * P) // 7}):
        check(dims, "allreduce", "B", ports, "BINE", ports * P * 3 + extra * ports + ports // 2)
    if ports == 1:
        check(dims, "allreduce", "B", 1, "RECDOUB", P * 5 + P // 3)


@pytest.mark.parametrize("dims,coll,variant,ports,family", [
    ([2048], "allreduce", "L", 1, "BINE"), ([8192], "allreduce", "L", 1, "RECDOUB"), ([2, 1024], "allreduce", "L", 4, "BINE"),
    ([128], "allgather", "VEC_DOUBLING_CONT_PERMUTE", 1, "BINE"), ([16, 8], "allgather", "VEC_DOUBLING_CONT_PERMUTE", 4, "BINE")])
def test_uniform_messages_match_the_host(dims, coll, variant, ports, family):
    check(dims, coll, variant, ports, family, 1001)
