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
