"""FP64 step kernels at the edges of their tile sizes: bit for bit with the CPU oracle.

The launch picks one of three tile sizes per degree from the mesh and the number of SMs;
the meshes below cover all three at every degree, with partly filled tiles on both axes,
more receivers than one sampling CTA takes, sources on element corners, and field values
whose quotients leave the range of the reciprocal-based division.
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


def _spec(mx, my, p, nrec):
    rng = np.random.default_rng(100 * mx + my + p)
    vp = rng.uniform(3000, 6000, mx * my)
    rec = [(float(x), float(y)) for x, y in rng.uniform(-990, 990, (nrec, 2))]
    return S.demo(mx, my, p=p, tmax=1.0e30).replace(
        nt=1000, cell_vp=vp, cell_vs=vp / 1.7, cell_rho=rng.uniform(2000, 3000, mx * my), receivers=rec,
        nearest_internal_gll=p > 1)


def _check(sp, steps, u, v, a):
    sol, ref = G.Solver(H.Setup(sp), "fp64"), O.OracleSolver(sp)
    sol.set_fields(u, v, a)
    ref.set_state(u, v, a)
    rows = [sol.run(n) for n in steps]
    want = ref.run(sum(steps))
    assert np.array_equal(np.concatenate(rows), want["traces"][:sum(steps)], equal_nan=True)
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(sol.fields(), ref.state()))
    return sol


@pytest.mark.parametrize("p", range(1, 9))
@pytest.mark.parametrize("nodes", [30, 4000, 60000])
def test_tile_sizes_match_the_oracle(p, nodes):
    mx, my = max(1, round(nodes ** 0.5 / p) + 1), max(1, round(0.9 * nodes ** 0.5 / p))
    sp = _spec(mx, my, p, 3 if nodes < 100 else 70)
    rng = np.random.default_rng(p)
    n = 2 * (mx * p + 1) * (my * p + 1)
    _check(sp, (1, 3), *(rng.standard_normal(n) * s for s in (1e-6, 1e-3, 1.0)))


@pytest.mark.parametrize("p", [2, 5])
def test_quotients_over_the_whole_range(p):
    """Accelerations from subnormal to near overflow, exact zeros of both signs among the fields."""
    sp = _spec(9, 7, p, 5)
    rng = np.random.default_rng(7)
    n = 2 * (9 * p + 1) * (7 * p + 1)
    scale = 10.0 ** rng.uniform(-320, 285, n)
    zero = np.where(rng.random(n) < 0.2, rng.choice([0.0, -0.0], n), 1.0)
    _check(sp, (2,), rng.standard_normal(n) * scale * zero, np.zeros(n), -np.zeros(n))
    # a quiet half: the wave front decays through the subnormal range into zeros
    u = np.zeros(n)
    u[:4] = 1e-300
    _check(sp, (3,), u, np.zeros(n), np.zeros(n))


@pytest.mark.parametrize("p", range(1, 9))
def test_force_matches_the_oracle(p):
    sp = _spec(11, 6, p, 1)
    sol, ref = G.Solver(H.Setup(sp), "fp64"), O.OracleSolver(sp)
    u = np.random.default_rng(p).standard_normal(2 * (11 * p + 1) * (6 * p + 1))
    assert np.array_equal(sol.assemble_linear_form(u), ref.force(u))
