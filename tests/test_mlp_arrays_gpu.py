"""The arrays that a caller hands to the picker MLP's training step."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine

pytestmark = pytest.mark.gpu


def batch(n, din, dout, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn((n, din), device="cuda", generator=g)
    t = torch.randn((n, dout), device="cuda", generator=g)
    mask = (torch.rand((n, dout), device="cuda", generator=g) < 0.5).float()
    return x, t, mask


@pytest.mark.parametrize("n,dout", [(16, 16), (256, 144)])
def test_arrays_may_be_overwritten_after_a_step_without_a_loss(n, dout):
    """A step called with no place for the loss has read its arrays when it
    returns: they are overwritten from another stream at once, with the
    step's own stream held up, and the parameters are those of steps that
    were waited for."""
    a, b = (bine.MLP(16, 256, dout, n, seed=5) for _ in range(2))
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    for step in range(4):
        arrays = batch(n, 16, dout, step)
        a.train_step(*arrays, 1e-3)
        torch.cuda.synchronize()
        with torch.cuda.stream(own):
            torch.cuda._sleep(4_000_000)
        x, t, mask = arrays
        b._check(bine.lib().bine_mlp_train_step(b._h, x.data_ptr(), t.data_ptr(), mask.data_ptr(), n, 1e-3,
                                                own.cuda_stream, None))
        with torch.cuda.stream(other):
            for v in arrays:
                v.fill_(float("nan"))
        torch.cuda.synchronize()
        assert np.array_equal(a.get_params(), b.get_params()), step
    a.close()
    b.close()


@pytest.mark.parametrize("n,dout", [(16, 16), (48, 144)])
def test_pinned_output_targets_and_mask(n, dout):
    """Arrays that are not the device's own memory go through copies of the
    runtime: the same bits as from device arrays."""
    m = bine.MLP(16, 256, dout, 64, seed=6)
    x, t, mask = batch(n, 16, dout, 1)
    y = torch.full((n, dout), -1.0).pin_memory()
    m._check(bine.lib().bine_mlp_forward(m._h, x.data_ptr(), n, y.data_ptr(), 0))
    torch.cuda.synchronize()
    assert torch.equal(y, m.forward(x).cpu())
    g, loss = m.gradients(x, t, mask)
    tp, mp = t.cpu().pin_memory(), mask.cpu().pin_memory()
    for tt, mm in ((tp, mp), (tp, mask), (t, mp)):
        g2, loss2 = m.gradients(x, tt, mm)
        assert np.array_equal(g, g2) and loss == loss2
    m.close()


def test_a_pageable_output_is_refused():
    """No kernel is launched on it."""
    m = bine.MLP(16, 16, 16, 16)
    x = torch.zeros((16, 16), device="cuda")
    y = np.full((16, 16), -1.0, np.float32)
    assert bine.lib().bine_mlp_forward(m._h, x.data_ptr(), 16, y.ctypes.data, 0) != bine.SUCCESS
    assert bine.lib().bine_mlp_forward(m._h, x.data_ptr(), 16, None, 0) != bine.SUCCESS
    torch.cuda.synchronize()
    assert (y == -1).all()
    m.close()


def test_a_batch_of_more_rows_of_tiles_than_a_grid_has_rows():
    """65,537 rows of 32-row tiles: the last rows are those of a small batch,
    and the loss is the mean over all of them."""
    n, last = 32 * 65537, 64
    m = bine.MLP(16, 16, 16, n, seed=7)
    x = torch.randn((n, 16), device="cuda")
    y = m.forward(x)
    assert torch.equal(y[-last:], m.forward(x[-last:].contiguous()))
    assert torch.equal(y[:last], m.forward(x[:last].contiguous()))
    t, mask = torch.zeros((n, 16), device="cuda"), torch.ones((n, 16), device="cuda")
    g, loss = m.gradients(x, t, mask)
    # 65,537 block partials in fp32, 2,049 to a lane, after the additions in
    # a block: fewer than 4,200 in a row, each rounding by at most 2^-24.
    assert abs(loss - float((y.double() ** 2).mean())) <= 4200 * 2.0 ** -24 * loss
    assert np.isfinite(g).all()
    m.close()
