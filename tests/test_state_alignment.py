"""The device state's arrays start on 256-byte boundaries, as allocations do, at every mesh size."""
import pytest

from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


@pytest.mark.parametrize("precision", ["fp64", "fp32_df", "fp32_kahan", "fp32"])
@pytest.mark.parametrize("mx,my,p", [(1, 1, 1), (5, 3, 2), (7, 9, 3), (13, 4, 8)])
def test_device_fields_are_aligned(mx, my, p, precision):
    sol = G.Solver(H.Setup(S.demo(mx, my, p=p, tmax=1e30).replace(nt=100, nearest_internal_gll=p > 1)), precision)
    for _ in range(2):
        assert all(x % 256 == 0 for x in sol.device_fields())
        sol.advance(1)   # (the other buffer set)
