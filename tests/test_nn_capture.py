"""Captured passes of the surrogate network: a graph made from a forward pass or an optimiser step
gives, when it is replayed, what the same calls give at that moment.

The GEMM path reads mode blocks formed from the parameters; they have to follow every change of
the parameters, eager or replayed, whatever ran or was captured before.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from se2dr_fork_gb300 import nn as N  # noqa: E402

pytestmark = pytest.mark.gpu

# width 80 has no fused kernels: the GEMM path in every mode
CASES = [(80, 1), (32, 0), (32, 2), (32, 1)]


@pytest.fixture(autouse=True)
def _built(nn_lib):
    yield nn_lib
    N.set_tensor_path(1)


class _Net:
    def __init__(self, width):
        self.c = N.Config(ny=16, nx=32, cin=16, width=width, modes=4, layers=2, nrec=4, nout=64, hidden=32, max_batch=2)
        self.net = N.Network(self.c, seed=3)
        self.net.set_receivers(np.arange(4) * 5)
        self.stream = torch.cuda.Stream()
        self.net.set_stream(self.stream.cuda_stream)
        g = torch.Generator(device="cuda").manual_seed(1)
        self.x = torch.randn(2, 16, 32, 16, generator=g, device="cuda").bfloat16()
        self.t = torch.randn(2, 4, 64, generator=g, device="cuda")
        self.out = torch.zeros(2, 4, 64, device="cuda")
        torch.cuda.synchronize()

    def capture(self, f):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=self.stream):
            f()
        return graph

    def replay(self, graph):
        with torch.cuda.stream(self.stream):
            graph.replay()
        torch.cuda.synchronize()

    def forward(self):
        self.net.forward(self.x, self.out)
        torch.cuda.synchronize()
        return self.out.cpu().numpy()

    def captured_forward(self):
        return self.capture(lambda: self.net.forward(self.x, self.out))


def _expected(width, params):
    """The forward pass of a new network with these parameters."""
    n = _Net(width)
    n.net.set_params(params)
    return n.forward()


@pytest.mark.parametrize("width,mode", CASES)
@pytest.mark.parametrize("ran_before", [False, True])
def test_captured_forward_follows_the_parameters(width, mode, ran_before):
    N.set_tensor_path(mode)
    n = _Net(width)
    if ran_before:
        n.forward()
    graph = n.captured_forward()
    assert np.array_equal(n.forward(), _expected(width, n.net.params()))   # (not yet replayed)
    rng = np.random.default_rng(5)
    for k in range(3):
        p = n.net.params() + 0.05 * rng.standard_normal(n.net.nparams).astype(np.float32)
        n.net.set_params(p)
        n.out.zero_()
        n.replay(graph)
        assert np.array_equal(n.out.cpu().numpy(), _expected(width, p)), k
        n.net.loss_grad(n.x, n.t)
        n.net.adam_step(1e-2)
        torch.cuda.synchronize()
        n.replay(graph)
        assert np.array_equal(n.out.cpu().numpy(), _expected(width, n.net.params())), k


@pytest.mark.parametrize("width,mode", CASES)
@pytest.mark.parametrize("ran_before", [False, True])
def test_replayed_optimiser_step_reaches_the_forward_pass(width, mode, ran_before):
    N.set_tensor_path(mode)
    n = _Net(width)
    n.net.loss_grad(n.x, n.t)
    if not ran_before:   # (gradients without the forward pass having run on this handle's blocks since)
        n.net.set_params(n.net.params())
    step = n.capture(lambda: n.net.adam_step(1e-2))
    for k in range(3):
        if k:
            n.forward()
        n.replay(step)
        assert np.array_equal(n.forward(), _expected(width, n.net.params())), k
