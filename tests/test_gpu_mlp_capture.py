"""A captured gradient follows the network's parameters: replayed after
set_params it is the gradient at the new parameters, and a capture that is
never replayed leaves later gradients alone.  Same kernels on the same values
as the eager call, so equality (the loss is summed by atomics and not
compared)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(seed, hidden):
    from ice3gb.mlp import Mlp
    return Mlp(16, hidden, 2, 10, seed=seed)


def _batch(n=200):
    rng = np.random.default_rng(n)
    t = np.zeros((n, 16), dtype=np.float32)
    t[:, 0:10:2] = rng.uniform(size=(n, 5)) < 0.5
    t[:, 1:10:2] = rng.standard_normal((n, 5))
    return torch.as_tensor(rng.standard_normal((n, 16)).astype(np.float32)).cuda(), torch.as_tensor(t).cuda()


def _capture(net, x, t):
    from ice3gb import _abi
    g = torch.zeros(net.n_params, dtype=torch.float32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _abi.check(net.lib.ice3gb_mlp_loss_grad(
            net.h, int(x.shape[0]), ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(t.data_ptr()),
            ctypes.c_void_p(g.data_ptr()), None, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), None, "capture")
    return graph, g


@pytest.mark.parametrize("hidden", [256, 40])
def test_replay_after_set_params(hidden):
    x, t = _batch()
    net, other = _net(1, hidden), _net(2, hidden)
    net.loss_grad(x, t)                                # allocates the workspaces
    graph, g = _capture(net, x, t)
    net.set_params(other.get_params())
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(g, other.loss_grad(x, t)[1])
    net.check()


@pytest.mark.parametrize("hidden", [256, 40])
def test_capture_without_replay(hidden):
    x, t = _batch()
    net, other = _net(1, hidden), _net(2, hidden)
    net.loss_grad(x, t)
    net.set_params(other.get_params())
    _capture(net, x, t)
    assert torch.equal(net.loss_grad(x, t)[1], other.loss_grad(x, t)[1])
    net.check()
