"""An ensemble with more chunks than launch chains: two chunks share a chain, in streams and in the
captured graph, and every shot still has the bits of a run of its own."""
import numpy as np
import pytest

from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(gpu_lib):
    return gpu_lib


def _shots():
    # 200 shots of degree 1 are three chunks of up to 96; the other degrees one each: ten chunks on
    # eight chains
    degrees = [1] * 200 + [2, 3, 4, 5, 6, 7, 8]
    out = []
    for i, p in enumerate(degrees):
        m = 3 + i % 4 if p == 1 else 6 + p
        out.append(H.Setup(S.shot(11, i, size=(m, m + 1), p=p, nt=40).replace(nearest_internal_gll=p > 1)))
    return out


@pytest.mark.parametrize("graphs", [False, True])
def test_ten_chunks_on_eight_chains(graphs):
    setups = _shots()
    ens = G.Ensemble(setups, "fp32_kahan", block=4)
    ens.set_graphs(graphs)
    rows = [ens.advance(n) for n in (8, 3, 9)]
    for i in [0, 1, 95, 96, 150, 191, 192, *range(199, 207)]:
        sol = G.Solver(setups[i], "fp32_kahan")
        want = sol.run(20)
        assert np.array_equal(np.concatenate([r[i] for r in rows]), want), i
        assert all(np.array_equal(x, y) for x, y in zip(ens.fields(i), sol.fields())), i
        sol.close()
