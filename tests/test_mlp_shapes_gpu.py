"""The picker MLP's layered kernels at the edges of their tiles: widths and
batches that do not fill a 32 x 32 tile, reductions longer than the two
staged buffers, masks with no valid entry.  Same reference and tolerances as
for the picker's own shape."""
import numpy as np
import pytest
import torch

import bine_trees_fugaku_b200 as bine
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("din,h,dout,n", [(16, 16, 16, 16), (48, 80, 16, 48), (16, 256, 144, 256), (32, 272, 304, 16),
                                          (64, 48, 16, 528), (272, 32, 48, 272)])
def test_gradients_and_forward_at_tile_edges(din, h, dout, n):
    rng = np.random.default_rng(din + h + n)
    m = bine.MLP(din, h, dout, n, seed=3)
    lay = bine.mlp_layout(din, h, dout)
    p = m.get_params()
    for w, b, nout, nin in lay:
        p[b:b + nout] = rng.standard_normal(nout).astype(np.float32) * 0.1
    m.set_params(p)
    x = rng.standard_normal((n, din)).astype(np.float32)
    t = rng.standard_normal((n, dout)).astype(np.float32)
    mask = (rng.random((n, dout)) < 0.4).astype(np.float32)
    mask[0, 0] = 1
    xd, td, md = (torch.from_numpy(a).cuda() for a in (x, t, mask))
    y = m.forward(xd).cpu().numpy()
    ref_y = mlp_ref.forward(p, lay, x)[0][-1]
    assert np.abs(y - ref_y).max() <= 2e-2 * np.abs(ref_y).max()
    g, loss = m.gradients(xd, td, md)
    ref_loss, ref_g = mlp_ref.loss_and_grads(p, lay, x, t, mask)
    assert abs(loss - ref_loss) <= 1e-3 * ref_loss
    for w, b, nout, nin in lay:
        for lo, hi in ((w, w + nout * nin), (b, b + nout)):
            a, r = g[lo:hi].astype(np.float64), ref_g[lo:hi]
            rel = np.linalg.norm(a - r) / max(1e-30, np.linalg.norm(r))
            assert rel < 2e-2, (lo, rel)
    # The same call again gives the same bits, the loss included.
    g2, loss2 = m.gradients(xd, td, md)
    assert np.array_equal(g, g2) and loss == loss2
    # A mask without a valid entry: no loss, no gradient.
    g0, loss0 = m.gradients(xd, td, torch.zeros_like(md))
    assert loss0 == 0 and not g0.any()
    m.close()


def test_host_targets_are_refused():
    m = bine.MLP(16, 16, 16, 16)
    x = torch.zeros((16, 16), device="cuda")
    with pytest.raises(bine.BineError):
        m.gradients(x, torch.zeros((16, 16)), x)
    m.close()
