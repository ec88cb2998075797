"""Which tiles a new handle runs, and that its configuration number names them."""
import numpy as np
import pytest

from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _solver(mx, my, p, precision):
    return G.Solver(H.Setup(S.demo(mx, my, p=p, tmax=1e30).replace(nt=100, nearest_internal_gll=p > 1)), precision)


# (degree, mesh edge, tile edge, threads, owned buffers) on 152 SMs, both sides of each line where
# other tiles than the degree's own take over, and the number that a new handle has
CHOICES = [
    ("fp32_kahan", 4, 9, 3, 192, 1, 1), ("fp32_kahan", 4, 71, 3, 192, 1, 1), ("fp32_kahan", 4, 77, 7, 320, 2, 1),
    ("fp32_kahan", 4, 128, 8, 416, 1, 1), ("fp32_kahan", 4, 260, 7, 320, 2, 1),
    ("fp32", 4, 128, 8, 416, 1, 1), ("fp32", 4, 260, 7, 320, 2, 1),
    ("fp32_kahan", 7, 20, 2, 256, 1, 2), ("fp32_kahan", 7, 85, 5, 288, 1, 2), ("fp32", 7, 85, 5, 288, 1, 2),
    ("fp32_kahan", 6, 20, 2, 192, 1, 0), ("fp32_kahan", 6, 47, 4, 192, None, 0), ("fp32_kahan", 6, 150, 5, 256, None, 0),
    ("fp32", 8, 150, 4, 256, None, 0), ("fp32_kahan", 8, 150, 3, 160, None, 1),
    ("fp32_df", 4, 60, 3, 192, 1, 0), ("fp32_df", 4, 250, 5, 128, 1, 0),
]


@pytest.mark.parametrize("precision,p,m,edge,threads,owned,number", CHOICES)
def test_new_handle_reports_the_tiles_it_runs(precision, p, m, edge, threads, owned, number):
    sol = _solver(m, m, p, precision)
    assert sol.tile_config == number
    assert sol.tile_configs()[number] == (edge, threads)
    info = sol.tile_config_info(number)
    assert (info["edge"], info["threads"]) == (edge, threads)
    assert owned is None or info["owned_buffers"] == owned
    # a block of n steps without a halo is n + 1 launches, with one n; selecting the reported number
    # again changes neither
    before = sol.info()["launches"]
    sol.advance(5)
    n = sol.info()["launches"] - before
    assert n == (6 if precision == "fp32_df" or edge * p <= 14 else 5)
    sol.set_tile_config(number)
    assert sol.tile_config == number
    before = sol.info()["launches"]
    sol.advance(5)
    assert sol.info()["launches"] - before == n


@pytest.mark.parametrize("p", range(1, 9))
def test_two_float_numbers_of_small_tiles_come_last(p):
    """A two-float number kept from another list of tiles selects one that a large mesh can run on:
    the tiles of small meshes are the last ones."""
    m = 1000 // p
    edges = [e for e, _ in _solver(m, m, p, "fp32_df").tile_configs()]
    assert min(edges) not in edges[:len(edges) // 2] and max(edges) in edges[:2]


@pytest.mark.parametrize("precision", ["fp32_kahan", "fp32"])
@pytest.mark.parametrize("p", range(1, 9))
def test_block_of_one_step_is_one_launch(p, precision):
    """On a small mesh a block of one step runs the tiles with a halo, unless the step without one
    was selected by its own number; the states and rows are those of any other block length."""
    m = 60 // p
    sol, ref, own = (_solver(m, m, p, precision) for _ in range(3))
    own.set_tile_config(len(own.tile_configs()) - 1)
    for s, launches in ((sol, 1), (own, 2)):
        before = s.info()["launches"]
        s.advance(1)
        assert s.info()["launches"] - before == launches
    sol.advance(3)
    for _ in range(3):
        sol.advance(1)
    own.advance(6)
    ref.advance(7)
    want = [ref.traces(), *ref.fields()]
    for s in (sol, own):
        assert all(np.array_equal(x, y) for x, y in zip([s.traces(), *s.fields()], want))
