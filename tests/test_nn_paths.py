"""Which kernels a surrogate pass runs on: the fused ones wherever the shape allows, GEMMs elsewhere."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from se2dr_fork_gb300 import nn as N  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _built(nn_lib):
    yield nn_lib
    N.set_tensor_path(1)


# ny, nx, cin, width, modes, nrec, nsub, hidden; are the layers fused, is the decoder
CASES = [
    ((8, 16, 16, 16, 1, 1, 2, 16), True, True),
    ((128, 128, 16, 64, 16, 16, 16, 128), True, True),
    ((40, 80, 64, 48, 9, 128, 8, 48), True, True),
    ((16, 32, 16, 32, 4, 4, 24, 32), True, False),      # outputs per row
    ((16, 32, 16, 32, 4, 4, 4, 144), True, False),      # hidden width
    ((12, 32, 16, 32, 4, 4, 4, 32), False, False),      # height
    ((136, 32, 16, 32, 4, 4, 4, 32), False, False),
    ((16, 144, 16, 16, 4, 4, 4, 32), False, False),     # width of the row
    ((16, 24, 16, 16, 4, 4, 4, 32), False, False),
    ((16, 32, 16, 80, 4, 4, 4, 32), False, False),      # channels
    ((16, 32, 80, 32, 4, 4, 4, 32), False, False),
    ((48, 48, 16, 32, 17, 4, 4, 32), False, False),     # modes
    ((16, 32, 16, 32, 4, 129, 4, 32), False, False),    # receivers
]


def _gemms(f):
    def total():
        i = N.tensor_path_info()
        return sum(v for v in i.values() if not isinstance(v, bool))
    a = total()
    f()
    torch.cuda.synchronize()
    return total() - a


@pytest.mark.parametrize("shape,layers,decoder", CASES)
def test_kernels_of_a_pass(shape, layers, decoder):
    ny, nx, cin, w, m, nrec, nsub, hidden = shape
    net = N.Network(N.Config(ny=ny, nx=nx, cin=cin, width=w, modes=m, layers=2, nrec=nrec, nout=ny * nsub, hidden=hidden, max_batch=2), seed=1)
    net.set_receivers(np.arange(nrec) % nx)
    x = torch.randn(2, ny, nx, cin, device="cuda").bfloat16()
    out, t = (torch.zeros(2, nrec, ny * nsub, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    N.set_tensor_path(0)
    every = _gemms(lambda: net.forward(x, out)), _gemms(lambda: net.loss_grad(x, t))
    N.set_tensor_path(1)
    now = _gemms(lambda: net.forward(x, out)), _gemms(lambda: net.loss_grad(x, t))
    if layers and decoder:
        assert now == (0, 0)
    elif layers:
        assert 0 < now[0] < every[0] and 0 < now[1] < every[1]   # the decoder's
    else:
        assert now == every and every[0] > 0
    # an input that is not 16-byte aligned: no fused layers
    y = torch.empty(x.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view_as(x).copy_(x)
    torch.cuda.synchronize()
    assert _gemms(lambda: net.forward(y, out)) == every[0]
