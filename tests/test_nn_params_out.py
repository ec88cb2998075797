"""Parameters and gradients into the caller's host array, whatever memory that is."""
import ctypes as C
import mmap

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from se2dr_fork_gb300 import nn as N  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(nn_lib):
    # 1.06 million parameters: 65 pages of 64 KB, 1040 of 4 KB
    n = N.Network(N.Config(ny=16, nx=32, cin=16, width=64, modes=4, layers=4, nrec=4, nout=64, hidden=32, max_batch=2), seed=3)
    n.set_params(np.random.default_rng(1).standard_normal(n.nparams).astype(np.float32))
    return n


def _get(net, a):
    assert a.size == net.nparams and a.dtype == np.float32
    assert N.lib().se2nn_get_params(net._h, a.ctypes.data_as(C.POINTER(C.c_float))) == 0


@pytest.mark.parametrize("offset", [0, 1, 3, 1024])   # floats into the memory
@pytest.mark.parametrize("kind", ["new", "used", "half", "pinned"])
def test_every_kind_of_host_memory(net, kind, offset):
    want, n = net.params(), net.nparams
    size = n + offset + 5
    if kind == "pinned":
        whole = torch.zeros(size, dtype=torch.float32).pin_memory().numpy()
    else:
        whole = np.frombuffer(mmap.mmap(-1, 4 * size), dtype=np.float32)   # (pages appear when they are touched)
    if kind == "used":
        whole[:] = 7.0
    if kind == "half":
        whole[:size // 3] = 7.0
    whole[:offset], whole[offset + n:] = -1.0, -2.0
    _get(net, whole[offset:offset + n])
    assert np.array_equal(whole[offset:offset + n], want)
    assert np.all(whole[:offset] == -1.0) and np.all(whole[offset + n:] == -2.0)


def test_copies_queued_before_read_the_array_as_it_was(net):
    """A copy out of the array, queued on the network's stream and not yet run, precedes the call."""
    want, stream = net.params(), torch.cuda.Stream()
    net.set_stream(stream.cuda_stream)
    pin = torch.randn(net.nparams).pin_memory()
    before, dev = pin.clone(), torch.zeros(net.nparams, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)   # 10 ms
        dev.copy_(pin, non_blocking=True)
        _get(net, pin.numpy())
    torch.cuda.synchronize()
    assert torch.equal(dev.cpu(), before)
    assert np.array_equal(pin.numpy(), want)


@pytest.mark.parametrize("call", ["se2nn_get_params", "se2nn_get_grads"])
def test_device_memory_is_not_stored_to_by_the_host(net, call):
    """A device pointer is the copy's to refuse or to serve: the host threads leave it alone."""
    dev = torch.full((net.nparams,), 5.0, device="cuda")
    torch.cuda.synchronize()
    rc = getattr(N.lib(), call)(net._h, C.cast(dev.data_ptr(), C.POINTER(C.c_float)))
    want = net.params() if call == "se2nn_get_params" else net.grads()
    assert np.array_equal(dev.cpu().numpy(), want if rc == 0 else np.full(net.nparams, 5.0, np.float32))


@pytest.fixture(scope="module")
def large(nn_lib):
    # 4.2 million parameters, 17 MB: several threads
    n = N.Network(N.Config(ny=16, nx=32, cin=16, width=64, modes=8, layers=4, nrec=4, nout=64, hidden=32, max_batch=2), seed=3)
    n.set_params(np.random.default_rng(1).standard_normal(n.nparams).astype(np.float32))
    return n


@pytest.mark.parametrize("offset", [0, 1, 1024])
@pytest.mark.parametrize("kind", ["new", "used", "half", "pinned"])
def test_large_arrays_of_every_kind_of_host_memory(large, kind, offset):
    assert large.nparams * 4 > 16e6
    test_every_kind_of_host_memory(large, kind, offset)


@pytest.mark.parametrize("call", ["se2nn_get_params", "se2nn_get_grads"])
def test_large_device_memory_is_not_stored_to_by_the_host(large, call):
    test_device_memory_is_not_stored_to_by_the_host(large, call)
