"""Tiles under a handle's other duties: many tiles per CTA at degree 7, a checkpoint that goes on
under another configuration.
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


def _setup(mx, my, p, te):
    """Receivers and sources on the lines between tiles of te elements, and anywhere."""
    rng = np.random.default_rng(mx + p)
    n = mx * my
    vp = rng.uniform(3000, 6000, n)
    hx, hy = 2000.0 / mx, 2000.0 / my
    at = [(-1000 + te * i * hx + 1e-3, -1000 + te * j * hy + 1e-3) for i, j in ((1, 1), (2, 5), (mx // te, my // te), (7, 3))]
    rec = [(min(x, 999.0), min(y, 999.0)) for x, y in at] + [(float(x), float(y)) for x, y in rng.uniform(-990, 990, (9, 2))]
    src = S.demo(mx, my, p=p).sources
    src = src + [S.Source(x, y, (1e9, 0.0, 0.0, -1e9), S.STF_RICKER, (0.0, 6.0, 1.0)) for x, y in rec[:3]]
    return H.Setup(S.demo(mx, my, p=p, tmax=1e30).replace(
        nt=1000, cell_vp=vp, cell_vs=vp / 1.7, cell_rho=rng.uniform(2000, 3000, n), receivers=rec, sources=src))


@pytest.mark.parametrize("precision", ["fp32_kahan", "fp32"])
def test_degree_7_many_tiles_per_cta(precision):
    """150 x 141 elements: up to 1140 tiles, several per CTA, through one region stage as well as
    two; every configuration and any split of the run gives the same bits."""
    su = _setup(150, 141, 7, 5)
    rng = np.random.default_rng(7)
    fields = [rng.standard_normal(su.ndof) * s for s in (1e-6, 1e-3, 1.0)]
    want = None
    ncfg = len(G.Solver(su, precision).tile_configs())
    assert ncfg >= 5
    for c in [None, *range(ncfg)]:
        for blocks in ((9,), (4, 1, 4)):
            sol = G.Solver(su, precision)
            if c is not None:
                sol.set_tile_config(c)
            elif precision == "fp32_kahan":
                assert sol.tile_configs()[sol.tile_config] == (5, 288)   # one stage
            sol.set_fields(*fields)
            got = [np.concatenate([sol.run(n) for n in blocks]), *sol.fields()]
            sol.close()
            want = got if want is None else want
            assert all(np.array_equal(x, y) for x, y in zip(got, want)), (c, blocks)


@pytest.mark.parametrize("precision", ["fp32_kahan", "fp32", "fp32_df"])
@pytest.mark.parametrize("p", [2, 3, 4, 7])
def test_checkpoint_goes_on_under_another_configuration(p, precision):
    """Saved under one configuration (with or without a halo, a receiver row pending), loaded into a
    handle with another."""
    su = _setup(23, 19, p, 4)
    ref = G.Solver(su, precision)
    rows = ref.run(9)
    want = [ref.run(5), *ref.fields()]
    n = len(ref.tile_configs())
    for c in range(n):
        a = G.Solver(su, precision)
        a.set_tile_config(c)
        assert np.array_equal(a.run(9), rows)
        blob = a.checkpoint()
        for d in range(n):
            b = G.Solver(su, precision)
            b.set_tile_config(d)
            b.restore(blob)
            assert all(np.array_equal(x, y) for x, y in zip([b.run(5), *b.fields()], want)), (c, d)
            b.close()
        a.close()
