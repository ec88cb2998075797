"""Each of the three FP64 tile sizes of every degree, bit for bit with the CPU oracle.

The launch takes the size with the least work on the busiest SM; the meshes below were chosen
with that rule for 152 SMs, one per size, partly filled tiles on both axes wherever tiles are
wider than an element, and the tile information says which size runs (at degree 6 the two wider ones differ in rows only).
"""
import numpy as np
import pytest

from oracle import oracle as O
from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


# degree: (mesh, elements of a tile along x, threads) per size
SIZES = {
    1: [(13, 11, 4, 32), (49, 47, 8, 128), (120, 121, 16, 256)],
    2: [(13, 10, 3, 32), (37, 37, 7, 128), (65, 62, 8, 288)],
    3: [(13, 10, 2, 32), (29, 31, 4, 128), (45, 47, 4, 256)],
    4: [(13, 10, 1, 32), (23, 20, 5, 128), (46, 47, 5, 256)],
    5: [(11, 9, 1, 64), (20, 23, 3, 224), (29, 31, 4, 288)],
    6: [(11, 9, 1, 64), (23, 20, 5, 256), (42, 40, 5, 256)],
    7: [(11, 9, 1, 64), (11, 14, 2, 128), (47, 49, 4, 256)],
    8: [(11, 9, 1, 96), (17, 18, 3, 256), (30, 31, 4, 256)],
}
CASES = [(p, size) for p in SIZES for size in range(3)]


def _make(p, size):
    mx, my, edge, threads = SIZES[p][size]
    rng = np.random.default_rng(100 * p + size)
    n = mx * my
    vp = rng.uniform(3000, 6000, n)
    rec = [(float(x), float(y)) for x, y in rng.uniform(-990, 990, (40, 2))]
    sp = S.demo(mx, my, p=p, tmax=1.0e30).replace(
        nt=1000, cell_vp=vp, cell_vs=vp / 1.7, cell_rho=rng.uniform(2000, 3000, n), receivers=rec,
        nearest_internal_gll=p > 1)
    sol, ref = G.Solver(H.Setup(sp), "fp64"), O.OracleSolver(sp)
    assert sol.tile_configs() == [(edge, threads)]
    info = sol.tile_config_info(0)
    assert (info["edge"], info["threads"]) == (edge, threads)
    return rng, sol, ref, 2 * (mx * p + 1) * (my * p + 1)


@pytest.mark.parametrize("p,size", CASES)
def test_steps(p, size):
    rng, sol, ref, n = _make(p, size)
    fields = [rng.standard_normal(n) * s for s in (1e-6, 1e-3, 1.0)]
    sol.set_fields(*fields)
    ref.set_state(*fields)
    rows = np.concatenate([sol.run(1), sol.run(3)])
    assert np.array_equal(rows, ref.run(4)["traces"][:4])
    assert all(np.array_equal(x, y) for x, y in zip(sol.fields(), ref.state()))


@pytest.mark.parametrize("p,size", CASES)
def test_force(p, size):
    rng, sol, ref, n = _make(p, size)
    u = rng.standard_normal(n)
    assert np.array_equal(sol.assemble_linear_form(u), ref.force(u))
