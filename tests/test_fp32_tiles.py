"""The FP32 steps at the edges of their tiles: partly filled tiles on both axes, meshes smaller
than a tile, sources and receivers on tile corners.

Every tile configuration, with and without a halo of elements, and every split of a run into
blocks gives the same bits (a node's arithmetic does not depend on either), and those of the
two-float mode agree with FP64: each of about 40 operations on
the way from u to a rounds at 2^-46 relative to its operands, the derivative sums cancel by two
orders of magnitude at the most, which over the few steps run here stays below 1e-10 of the
largest value.
"""
import numpy as np
import pytest

from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _run(su, precision, blocks, fields, config=None):
    sol = G.Solver(su, precision)
    if config is not None:
        sol.set_tile_config(config)
    sol.set_fields(*fields)
    rows = np.concatenate([sol.run(n) for n in blocks])
    return [rows, *sol.fields()]


@pytest.mark.parametrize("p", range(1, 9))
@pytest.mark.parametrize("mx,my", [(1, 1), (2, 17), (13, 5), (25, 24), (61, 2)])
@pytest.mark.parametrize("precision", ["fp32_df", "fp32_kahan", "fp32"])
def test_tiles_and_blocks(p, mx, my, precision):
    rng = np.random.default_rng(1000 * p + 10 * mx + my)
    n = mx * my
    vp = rng.uniform(3000, 6000, n)
    rec = [(float(x), float(y)) for x, y in rng.uniform(-990, 990, (9, 2))]
    su = H.Setup(S.demo(mx, my, p=p, tmax=1.0e30).replace(
        nt=1000, cell_vp=vp, cell_vs=vp / 1.7, cell_rho=rng.uniform(2000, 3000, n), receivers=rec,
        nearest_internal_gll=p > 1))
    fields = [rng.standard_normal(su.ndof) * s for s in (1e-6, 1e-3, 1.0)]
    want = _run(su, precision, (4,), fields)
    for blocks in ((1, 3), (1, 1, 2)):
        assert all(np.array_equal(x, y) for x, y in zip(_run(su, precision, blocks, fields), want)), blocks
    for c in range(len(G.Solver(su, precision).tile_configs())):
        assert all(np.array_equal(x, y) for x, y in zip(_run(su, precision, (2, 2), fields, c), want)), c
    if precision != "fp32_df":
        return
    for x, y in zip(want, _run(su, "fp64", (4,), fields)):
        cols = np.abs(y).max(axis=0) if y.ndim > 2 else np.abs(y).max()
        assert np.all(np.abs(x - y) <= 1e-10 * np.maximum(cols, np.finfo(float).tiny))
