"""The training pass at the edges of its tiles: batches around one 128-row tile
and one weight-gradient range of 256 rows, hidden widths that are not multiples
of the 16-byte copies, every output width's padding.  Gradients against the
FP64 restatement with the kernels' BF16 roundings: an activation whose FP32 sum
differs in its last bit may round to the neighbouring BF16 value (2^-8 of it);
with a few per cent of them the relative norm stays below 2^-8 * 0.25 = 1e-3 per
layer, taken ten times for the layers above it."""
import mlp_ref
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, hidden, layers, n_out, seed):
    from ice3gb.mlp import Mlp
    net = Mlp(16, hidden, layers, n_out, seed=seed)
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, 16)).astype(np.float32)
    t = np.zeros((n, 16), dtype=np.float32)
    t[:, 0:n_out:2] = rng.uniform(size=(n, n_out // 2)) < 0.6
    t[:, 1:n_out:2] = rng.standard_normal((n, n_out // 2))
    return net, torch.as_tensor(x).cuda(), torch.as_tensor(t).cuda()


@pytest.mark.parametrize("n,hidden,layers,n_out", [(1, 256, 3, 10), (127, 256, 3, 10), (128, 256, 1, 16), (129, 40, 2, 4),
                                                   (255, 100, 3, 2), (257, 256, 2, 8), (513, 24, 1, 14)])
def test_gradients_at_tile_edges(n, hidden, layers, n_out):
    net, x, t = _case(n, hidden, layers, n_out, seed=n)
    net.loss_grad(x.repeat(3, 1), t.repeat(3, 1))      # a larger batch before: stale rows behind this one
    loss, g = net.loss_grad(x, t)
    net.check()
    lr, gr = mlp_ref.loss_grad(net.get_params(), net.layout(), x.cpu().numpy(), t.cpu().numpy())
    assert abs(loss - lr) <= 1e-3 * abs(lr)
    g = g.cpu().numpy().astype(np.float64)
    for wo, bo, o, i in net.layout():
        for lo, hi in ((wo, wo + o * i), (bo, bo + o)):
            assert np.linalg.norm(g[lo:hi] - gr[lo:hi]) <= 1e-2 * np.linalg.norm(gr[lo:hi])


def test_transposed_weights_follow_training_steps():
    """A training step refreshes the transposed weights itself; a network that
    is given the same parameters builds them anew: the same gradients."""
    net, x, t = _case(300, 256, 3, 10, seed=3)
    for _ in range(3):
        net.train_step(x, t, 1e-2)
    other, _, _ = _case(300, 256, 3, 10, seed=4)
    other.set_params(net.get_params())
    assert torch.equal(net.loss_grad(x, t)[1], other.loss_grad(x, t)[1])


@pytest.mark.parametrize("n,hidden,layers,n_out", [(129, 128, 2, 10), (200, 132, 2, 10), (257, 144, 3, 16), (130, 200, 2, 6),
                                                   (64, 252, 2, 2)])
def test_gradients_at_column_tile_edges(n, hidden, layers, n_out):
    """Hidden widths around the 128 columns of a CTA's tile, with a second tile
    from 4 columns to almost full; the bounds above."""
    test_gradients_at_tile_edges(n, hidden, layers, n_out)
