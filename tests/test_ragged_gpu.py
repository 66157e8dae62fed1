"""Rows and blocks off the 16-byte grid on the FUSED engine: packed rows of
odd length, blocks of odd length, buffers that start in the middle of a
vector.  Results are compared bit for bit with the oracle (floats in the
reference's order) or with exact sums and copies, and the bytes around the
receive rows stay as they were."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle import port
from oracle.common import buffer_counts, expected

pytestmark = pytest.mark.gpu

CODE = {np.dtype(np.int32): bine.INT32, np.dtype(np.int64): bine.INT64, np.dtype(np.float32): bine.FLOAT,
        np.dtype(np.float64): bine.DOUBLE, np.dtype(np.int8): bine.CHAR}
GUARD = 64  # elements before and after the receive rows


def values(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    if np.dtype(dtype).kind == "f":
        return rng.standard_normal(shape).astype(dtype)
    lim = 100 if dtype == np.int8 else 1000
    return rng.integers(-lim, lim + 1, shape).astype(dtype)


def call(coll, x, count, shift=0, pad=0, variant=None, lanes=0, order="reference", root=0):
    """The collective on rows `pad` elements longer than their data, in
    buffers that start `shift` elements after a 16-byte boundary; checks the
    guards and the padding."""
    P = x.shape[0]
    si, so = x.shape[1], buffer_counts(coll, count, P)[1]
    td = torch.from_numpy(x[:1, :1]).dtype
    comm = bine.Comm(P)
    if variant:
        comm.set_algo(coll, variant)
    comm.set_tree_split(lanes)
    comm.set_float_order(order)
    comm.set_stream(torch.cuda.current_stream())
    es = x.dtype.itemsize
    send = torch.zeros(P * (si + pad) + shift + 1, dtype=td, device="cuda")
    rows = send[shift:shift + P * (si + pad)].view(P, si + pad)
    rows[:, :si] = torch.from_numpy(x).cuda()
    recv = torch.full((P * (so + pad) + 2 * GUARD + shift,), 77, dtype=td, device="cuda")
    out = recv[GUARD + shift:GUARD + shift + P * (so + pad)].view(P, so + pad)
    if coll == "bcast":
        out[root, :so] = rows[root, :si]
    if pad:
        comm.set_layout((si + pad) * es, (so + pad) * es)
    comm.run(coll, rows, out, count, CODE[x.dtype], root)
    comm.synchronize()
    got = out[:, :so].cpu().numpy()
    assert (out[:, so:] == 77).all()
    assert (recv[:GUARD + shift] == 77).all() and (recv[GUARD + shift + P * (so + pad):] == 77).all()
    comm.close()
    return got


def same_bits(a, b):
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("P,count,shift,pad", [
    (4, 4, 1, 0), (6, 127, 0, 0), (16, 129, 0, 0), (16, 16 * 128 + 3, 1, 0), (24, 24 * 33 + 1, 0, 0),
    (48, 48 * 129 - 1, 1, 0), (96, 96 * 257 + 5, 0, 0), (130, 130 * 40 + 7, 0, 3), (64, 64 * 512, 1, 1), (256, 256 * 21 + 1, 0, 0),
    (520, 520 * 5 + 3, 0, 0)])
def test_exact_order_allreduce_matches_the_oracle(P, count, shift, pad, dtype):
    x = values((P, count), dtype, P + count)
    want, _ = port.run("allreduce", x, count, variant="B")
    assert same_bits(call("allreduce", x, count, shift, pad), want)


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("P,count", [(64, 64 * 130 + 1), (96, 96 * 600 + 3)])
def test_every_lane_count_gives_the_same_bits(P, count, lanes):
    x = values((P, count), np.float32, lanes)
    want, _ = port.run("allreduce", x, count, variant="B")
    assert same_bits(call("allreduce", x, count, lanes=lanes), want)


def test_per_rank_trees_off_the_grid():
    """The L butterfly's trees differ from rank to rank: one destination row
    per segment."""
    x = values((16, 259), np.float32, 3)
    want, _ = port.run("allreduce", x, 259, variant="L")
    assert same_bits(call("allreduce", x, 259, variant="L"), want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("P,count,shift", [(4, 1, 0), (8, 3, 1), (16, 33, 0), (64, 129, 0), (64, 1025, 1), (128, 17, 0)])
def test_exact_order_reduce_scatter_matches_the_oracle(P, count, shift, dtype):
    if dtype == np.float64:  # the reference reduces no 64-bit types here: whole numbers, exact in any order
        x = values((P, P * count), np.int32, P + count).astype(dtype)
        want = expected("reduce_scatter", x, P, count)
    else:
        x = values((P, P * count), dtype, P + count)
        want, _ = port.run("reduce_scatter", x, count)
    assert same_bits(call("reduce_scatter", x, count, shift), want)


@pytest.mark.parametrize("P,count,root", [(16, 1001, 0), (64, 64 * 65 + 3, 0)])
def test_exact_order_reduce_matches_the_oracle(P, count, root):
    x = values((P, count), np.float32, P)
    want, _ = port.run("reduce", x, count, root=root)
    assert same_bits(call("reduce", x, count, root=root)[root], want[root])


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.int8, np.float64])
@pytest.mark.parametrize("coll", ["allreduce", "reduce", "reduce_scatter"])
@pytest.mark.parametrize("P,count,shift,pad", [
    (2, 1, 0, 0), (3, 5, 1, 0), (7, 1025, 0, 0), (15, 4099, 1, 1), (16, 33, 0, 0), (33, 257, 0, 0), (97, 1031, 0, 2), (200, 3, 0, 0),
    (64, 2047, 0, 1), (520, 13, 0, 0)])
def test_sums_off_the_grid(coll, P, count, shift, pad, dtype):
    """Whole-number sums (FAST order for float64), with ragged tails on rows
    that are and are not on the 16-byte grid."""
    si, _ = buffer_counts(coll, count, P)
    x = values((P, si), np.int32 if dtype == np.float64 else dtype, P * 7 + count).astype(dtype)
    want = expected(coll, x, P, count, 0)
    got = call(coll, x, count, shift, pad, order="fast")
    rows = [0] if coll == "reduce" else slice(None)
    assert np.array_equal(got[rows], want[rows])


@pytest.mark.parametrize("P,count", [(33, 1027), (200, 65)])
def test_fast_float_sums_off_the_grid(P, count):
    """FP64 accumulation, one rounding: within half an ulp of the FP64 sum
    and that sum's own P 2^-52 sum|x|."""
    x = values((P, count), np.float32, P)
    want = x.astype(np.float64).sum(0)
    got = call("allreduce", x, count, order="fast")
    bound = np.abs(want) * 2.0 ** -24 + P * 2.0 ** -52 * np.abs(x).astype(np.float64).sum(0)
    assert np.all(np.abs(got - want) <= bound)
    # A last partial vector on rows that are on the grid: same bound.
    got = call("allreduce", x, count, pad=4 - count % 4, order="fast")
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("dtype", [np.int8, np.int32, np.int64])
@pytest.mark.parametrize("coll", ["alltoall", "scatter", "gather"])
@pytest.mark.parametrize("P,count,shift,pad", [
    (2, 1, 0, 0), (5, 3, 1, 0), (7, 16, 1, 0), (16, 17, 0, 1), (33, 64, 0, 0), (9, 255, 3, 0), (6, 257, 1, 2), (12, 1021, 0, 0),
    (8, 2047, 1, 0), (8, 2049, 3, 5), (5, 4096, 0, 0), (4, 10_001, 1, 1), (64, 40, 0, 4)])
def test_block_copies_off_the_grid(coll, P, count, shift, pad, dtype):
    """Blocks from one element to several pieces of a warp, at every kind of
    offset between source and destination."""
    root = P // 2
    si, _ = buffer_counts(coll, count, P)
    x = values((P, si), dtype, P + count)
    want = expected(coll, x, P, count, root)
    got = call(coll, x, count, shift, pad, root=root)
    rows = [root] if coll == "gather" else slice(None)
    assert np.array_equal(got[rows], want[rows])


@pytest.mark.parametrize("dtype", [np.int8, np.int32, np.int64])
@pytest.mark.parametrize("coll,P,count,shift,pad", [
    ("bcast", 3, 1, 0, 0), ("bcast", 16, 131_073, 1, 0), ("bcast", 17, 130_003, 0, 1), ("bcast", 40, 65_540, 1, 0),
    ("bcast", 200, 11_003, 0, 0), ("bcast", 33, 4096, 0, 0),
    ("allgather", 3, 5, 1, 0), ("allgather", 48, 1001, 0, 0), ("allgather", 48, 1001, 1, 3), ("allgather", 130, 129, 0, 0),
    ("allgather", 16, 8200, 0, 1), ("allgather", 37, 64, 0, 0)])
def test_broadcasts_off_the_grid(coll, P, count, shift, pad, dtype):
    """Below and above the size from which tiles are staged for bulk copies;
    rows at every offset within 16 bytes, packed and padded sources."""
    root = P // 3
    si, _ = buffer_counts("allreduce" if coll == "bcast" else coll, count, P)
    x = values((P, si), dtype, P + count)
    want = expected(coll, x, P, count, root)
    assert np.array_equal(call(coll, x, count, shift, pad, root=root), want)


@pytest.mark.parametrize("coll,P,count", [
    ("bcast", 56, 4 * 37_889), ("bcast", 56, 4 * (37_889 + 33)), ("bcast", 56, 4 * 50_000 + 4), ("bcast", 300, 4 * 20_001),
    ("bcast", 70, 4 * 30_003), ("allgather", 65, 4 * 600), ("allgather", 40, 4 * 1400), ("allgather", 300, 4 * 37), ("allgather", 96, 4 * 333)])
def test_large_broadcasts_on_the_grid(coll, P, count):
    """From 32 MiB written: one warp per block with one and two vectors per
    thread, 64 and 256 threads; the last warp partly filled."""
    x = torch.randint(-1000, 1001, (P, count), dtype=torch.int32, device="cuda", generator=torch.Generator("cuda").manual_seed(P))
    so = count * (P if coll == "allgather" else 1)
    out = torch.full((P * so + 2 * GUARD,), 77, dtype=torch.int32, device="cuda")
    y = out[GUARD:GUARD + P * so].view(P, so)
    comm = bine.Comm(P)
    comm.set_stream(torch.cuda.current_stream())
    if coll == "bcast":
        y[3] = x[3]
    comm.run(coll, x, y, count, bine.INT32, 3)
    comm.synchronize()
    want = x.reshape(-1) if coll == "allgather" else x[3]
    assert bool((y == want).all())
    assert bool((out[:GUARD] == 77).all()) and bool((out[GUARD + P * so:] == 77).all())
    comm.close()
