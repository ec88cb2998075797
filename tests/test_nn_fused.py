"""The surrogate's fused layer kernels against the GEMM path: the same bits.

se2nn_set_tensor_path(0) runs every contraction as a GEMM launch; the default runs the fused
kernels wherever the shape allows.  Both round to BF16 at the same places and accumulate in
the same order, so outputs, losses, gradients and updated weights are equal bit for bit at
every width, at partly filled tiles, k steps and sample groups, and for receivers that share
a column.  Shapes the fused kernels do not take fall back and stay unchanged.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from se2dr_fork_gb300 import nn as N  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(nn_lib):
    yield nn_lib
    N.set_tensor_path(1)


CASES = [
    # ny, nx, cin, width, modes, layers, nrec, nsub, hidden, batch
    (8, 16, 16, 16, 1, 1, 1, 2, 16, 1),
    (16, 32, 16, 16, 3, 2, 17, 3, 32, 3),
    (24, 48, 32, 32, 12, 3, 5, 16, 16, 33),
    (40, 80, 16, 48, 9, 2, 16, 8, 48, 5),
    (64, 112, 64, 64, 16, 2, 16, 16, 128, 2),
    (128, 128, 16, 64, 16, 4, 16, 16, 128, 3),
    (96, 96, 16, 48, 12, 3, 16, 16, 128, 34),
    # the decoder not fused: outputs per row, hidden width
    (16, 32, 16, 32, 4, 2, 4, 24, 32, 2),
    (16, 32, 16, 32, 4, 2, 4, 4, 144, 2),
    # not fused: height, width of the row, channels
    (12, 32, 16, 32, 4, 2, 4, 4, 32, 2),
    (16, 144, 16, 16, 4, 2, 4, 4, 32, 2),
    (16, 32, 16, 80, 4, 2, 4, 4, 32, 2),
]


def _train(path, cfg, rec, x, t, steps):
    N.set_tensor_path(path)
    net = N.Network(cfg, seed=3)
    net.set_receivers(rec)
    got = []
    for _ in range(steps):
        out = torch.zeros(x.shape[0], cfg.nrec, cfg.nout, device="cuda")
        got.append(net.loss_grad(x, t, out))
        got += [net.grads(), out.cpu().numpy()]
        net.adam_step(1e-3)
    out = torch.zeros(x.shape[0], cfg.nrec, cfg.nout, device="cuda")
    net.forward(x, out)
    torch.cuda.synchronize()
    return got + [net.params(), out.cpu().numpy()]


@pytest.mark.parametrize("case", CASES)
def test_fused_layers_are_bitwise_the_gemm_path(case):
    ny, nx, cin, w, m, layers, nrec, nsub, hidden, batch = case
    cfg = N.Config(ny=ny, nx=nx, cin=cin, width=w, modes=m, layers=layers, nrec=nrec, nout=ny * nsub, hidden=hidden, max_batch=batch + 1)
    g = torch.Generator(device="cuda").manual_seed(ny + nx + w)
    x = torch.randn(batch, ny, nx, cin, generator=g, device="cuda").bfloat16()
    t = torch.randn(batch, nrec, cfg.nout, generator=g, device="cuda")
    rec = np.random.default_rng(1).integers(0, nx, nrec)
    rec[-1] = rec[0]   # two receivers of one column
    torch.cuda.synchronize()
    a, b = (_train(path, cfg, rec, x, t, 2) for path in (0, 1))
    assert all(np.array_equal(p, q) for p, q in zip(a, b))
    # inputs that are not 16-byte aligned take the GEMM path
    y = torch.empty(x.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view_as(x).copy_(x)
    torch.cuda.synchronize()
    c = _train(1, cfg, rec, y, t, 1)
    assert np.array_equal(c[1], a[1]) and np.array_equal(c[2], a[2])
