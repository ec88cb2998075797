"""Host logic of the tile autotuner's measurement (no GPU): configurations that fail to set up."""
import pytest

from se2dr_fork_gb300 import autotune as A
from se2dr_fork_gb300 import gpu as G
from se2dr_fork_gb300 import host as H
from se2dr_fork_gb300 import spec as S


class FakeSolver:
    """The part of gpu.Solver that the measurement uses."""

    def __init__(self, setup, precision, trace_capacity=0):
        self.setup, self.precision = setup, G.PRECISIONS[precision]

    def tile_configs(self):
        return [(7, 320), (7, 320), (6, 256)]

    def tile_config_info(self, c):
        return {"edge": self.tile_configs()[c][0]}

    def close(self):
        pass


def _tune(monkeypatch, errors):
    def time_config(sol, c, steps):
        if c in errors:
            raise G.GpuError("se2gpu_set_tile_config failed", errors[c])
        return 3.0 - c

    monkeypatch.setattr(A, "Solver", FakeSolver)
    monkeypatch.setattr(A, "time_config", time_config)
    return A.tune(H.Setup(S.explosion64(16, 12, p=4)), write=False)


def test_a_configuration_that_does_not_fit_is_left_out(monkeypatch):
    res = _tune(monkeypatch, {2: G.ERR_NOMEM})
    assert res["config"] == 1 and [x["seconds"] for x in res["all"]] == [3.0, 2.0, None]


def test_another_failure_is_raised(monkeypatch):
    with pytest.raises(G.GpuError) as e:
        _tune(monkeypatch, {0: -2})
    assert e.value.code == -2


def test_a_cached_number_of_other_tiles_is_not_used(tmp_path, monkeypatch):
    monkeypatch.setattr(A, "CACHE", str(tmp_path / "tuning.json"))
    sol = FakeSolver(H.Setup(S.explosion64(16, 12, p=4)), "fp32_df")
    sol.selected = None
    sol.set_tile_config = lambda c: setattr(sol, "selected", c)
    for edge, threads, want in [(5, 128, None), (6, 224, None), (6, 256, 2)]:
        A.save({A.key(sol.setup, "fp32_df"): {"config": 2, "edge": edge, "threads": threads}})
        assert A.apply(sol) == (want or 0) and sol.selected == want
