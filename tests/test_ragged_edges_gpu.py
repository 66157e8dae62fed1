"""Calls on either side of the lines between the kernels for rows and blocks
off the 16-byte grid, against exact sums and copies; exact-order sums in place
and of infinities, NaNs and zeros."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle import port
from oracle.common import buffer_counts, expected
from tests.test_ragged_gpu import CODE, call, same_bits, values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coll", ["allreduce", "reduce", "reduce_scatter"])
@pytest.mark.parametrize("P", [15, 16])
@pytest.mark.parametrize("count,shift,pad", [(1, 0, 0), (1027, 1, 0), (1026, 0, 2)])
def test_sums_below_and_from_16_ranks(coll, P, count, shift, pad):
    """One element per thread below 16 ranks, strided vectors from there on;
    float32 in the FAST order: FP64 accumulation and one rounding, within half
    an ulp of the FP64 sum and that sum's own P 2^-52 sum|x|."""
    si, _ = buffer_counts(coll, count, P)
    rows = [0] if coll == "reduce" else slice(None)
    x = values((P, si), np.int64, P + count)
    assert np.array_equal(call(coll, x, count, shift, pad)[rows], expected(coll, x, P, count, 0)[rows])
    x = values((P, si), np.float32, P + count)
    want = expected(coll, x.astype(np.float64), P, count, 0)[rows]
    absum = expected(coll, np.abs(x).astype(np.float64), P, count, 0)[rows]
    got = call(coll, x, count, shift, pad, order="fast")[rows]
    assert np.all(np.abs(got - want) <= np.abs(want) * 2.0 ** -24 + P * 2.0 ** -52 * absum)


@pytest.mark.parametrize("dtype", [np.int8, np.int32, np.int64, np.float64])
@pytest.mark.parametrize("P,vectors", [(2, 1), (17, 1), (768, 1), (64, 16), (5, 1031)])
def test_reduce_scatter_of_whole_vectors(P, vectors, dtype):
    """Blocks of one vector to several tiles on the 16-byte grid: every vector
    at its owner's place."""
    count = vectors * 16 // np.dtype(dtype).itemsize
    x = values((P, P * count), np.int8, P + vectors).astype(dtype)
    assert np.array_equal(call("reduce_scatter", x, count, pad=0, order="fast"), expected("reduce_scatter", x, P, count))


@pytest.mark.parametrize("dtype,count,shift", [
    (np.int8, 4093, 1), (np.int8, 4096, 1), (np.int8, 4097, 0), (np.int32, 4096, 1), (np.int32, 4097, 0), (np.int32, 16384, 0),
    (np.int32, 16388, 0), (np.int64, 4096, 1), (np.int64, 4097, 0)])
@pytest.mark.parametrize("coll,P", [("scatter", 64), ("gather", 64), ("alltoall", 8)])
def test_block_copies_around_262144_elements(coll, P, dtype, count, shift):
    """64 blocks each: at and below 262,144 elements of the widest type that
    fits the call one per thread, above pieces or realigned vectors."""
    root = P - 1
    si, _ = buffer_counts(coll, count, P)
    x = values((P, si), dtype, count)
    rows = [root] if coll == "gather" else slice(None)
    assert np.array_equal(call(coll, x, count, shift, root=root)[rows], expected(coll, x, P, count, root)[rows])


@pytest.mark.parametrize("dtype", [np.int8, np.int32, np.int64])
@pytest.mark.parametrize("count,shift", [(15, 1), (16, 1), (17, 1), (33, 0)])
def test_many_short_blocks(dtype, count, shift):
    """Above 262,144 elements, on either side of 16 elements per block."""
    P = 160
    x = values((P, P * count), dtype, count)
    assert np.array_equal(call("alltoall", x, count, shift), expected("alltoall", x, P, count))


@pytest.mark.parametrize("coll,P,count,shift", [
    ("bcast", 16, 262_137, 1), ("bcast", 16, 262_147, 0), ("bcast", 512, 8193, 0), ("allgather", 64, 1023, 1),
    ("allgather", 64, 1025, 0), ("allgather", 33, 3851, 1), ("allgather", 33, 3853, 0)])
def test_broadcasts_around_16_mib(coll, P, count, shift):
    """int32 rows that are stored element by element below, and staged for bulk
    copies from there on."""
    si, _ = buffer_counts("allreduce" if coll == "bcast" else coll, count, P)
    x = values((P, si), np.int32, P + count)
    assert np.array_equal(call(coll, x, count, shift, root=P - 1), expected(coll, x, P, count, P - 1))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("P,count,lanes", [(4, 1, 0), (24, 2051, 0), (96, 4097, 2), (64, 1027, 8), (200, 601, 0)])
def test_exact_order_allreduce_in_place_off_the_grid(P, count, lanes, dtype):
    """Input and output are one array of packed rows of odd length."""
    if count < P:  # the bandwidth-optimal schedule needs a block per rank
        count += P
    x = values((P, count), dtype, P + count)
    want, _ = port.run("allreduce", x, count, variant="B")
    buf = torch.from_numpy(x).cuda()
    comm = bine.Comm(P)
    comm.set_algo("allreduce", "B")
    comm.set_tree_split(lanes)
    comm.set_stream(torch.cuda.current_stream())
    comm.allreduce(buf, buf, count, CODE[np.dtype(dtype)])
    comm.synchronize()
    assert same_bits(buf.cpu().numpy(), want)
    comm.close()


@pytest.mark.parametrize("engine", ["fused", "pipelined"])
@pytest.mark.parametrize("P,count,lanes", [(16, 131, 0), (24, 67, 0), (96, 389, 4), (64, 256, 0)])
def test_infinities_nans_and_signed_zeros(P, count, lanes, engine):
    """Columns of infinities of one and of both signs, a NaN, and zeros of
    either sign only: the reference's order gives the same class of result,
    and the same bits where it is a number."""
    x = values((P, count), np.float32, P)
    x[P // 2, 0::7] = np.inf
    x[P - 1, 1::7] = -np.inf
    x[0, 2::7], x[P // 3, 2::7] = np.inf, -np.inf
    x[1, 3::7] = np.nan
    x[:, 4::7] = -0.0
    x[:, 5::7] = 0.0
    x[::2, 5::7] = -0.0
    with np.errstate(invalid="ignore"):
        want, _ = port.run("allreduce", x, count, variant="B")
    comm = bine.Comm(P)
    comm.set_algo("allreduce", "B")
    comm.set_engine(engine)
    comm.set_tree_split(lanes)
    comm.set_stream(torch.cuda.current_stream())
    send = torch.from_numpy(x).cuda()
    recv = torch.zeros_like(send)
    comm.allreduce(send, recv, count, bine.FLOAT)
    comm.synchronize()
    got = recv.cpu().numpy()
    comm.close()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(want[:, 2::7]).all()
    assert np.array_equal(got.view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])


@pytest.mark.parametrize("coll,P", [("allreduce", 40), ("allreduce", 41), ("reduce", 24), ("reduce", 25),
                                    ("reduce_scatter", 24), ("reduce_scatter", 25)])
@pytest.mark.parametrize("extra", [-2, 3])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_sums_of_few_ranks_around_65536_elements(coll, P, extra, dtype):
    """One element per thread above 65,536 elements up to 40 (24) ranks,
    strided vectors below and beyond."""
    count = 65536 + extra if coll != "reduce_scatter" else 65536 // P + extra
    si, _ = buffer_counts(coll, count, P)
    x = values((P, si), dtype, P + extra)
    rows = [0] if coll == "reduce" else slice(None)
    assert np.array_equal(call(coll, x, count, 1)[rows], expected(coll, x, P, count, 0)[rows])
