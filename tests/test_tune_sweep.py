"""What tune.autotune_batch sweeps (no GPU: a stand-in batch records the candidates): where the
batch is solved in clusters, the options that only the grid-wide solver reads are neither tried nor
returned."""
import importlib
from types import SimpleNamespace

import numpy as np
import pytest


@pytest.fixture
def tune():
    return importlib.import_module("g-slam_on_gpu_and_fpga_b200.tune")


def _run(tune, monkeypatch, clusters, candidates=None, **opts):
    """Best candidate, timings and the options of every batch built, for a batch that is in clusters at
    the windows in `clusters`; the time falls with the window and the thread count."""
    built = []

    class Batch:
        def __init__(self, o):
            self.o, self.in_clusters = o, o["sell_window"] in clusters

        @classmethod
        def from_se2_list(cls, graphs, lams, **o):
            built.append(o)
            return cls(o)

        def round_all(self):
            return [SimpleNamespace(solve_ms=1.0 / (self.o["sell_window"] + self.o["threads_per_cta"]))]

        def close(self):
            pass

    monkeypatch.setattr(tune, "PoseGraphBatch", Batch)
    graph = SimpleNamespace(init=np.zeros((3, 3)), edge_i=np.zeros(2))
    best, timings = tune.autotune_batch([graph], [0.1], candidates=candidates, **opts)
    return best, timings, built


def test_clusters_sweep_the_window_alone(tune, monkeypatch):
    best, timings, built = _run(tune, monkeypatch, clusters={32, 256, 1024})
    assert best == {"sell_window": 1024}
    assert [c for c, _ in timings] == [{"sell_window": w} for w in (32, 256, 1024)]
    assert len(built) == 3


def test_grid_wide_sweeps_everything(tune, monkeypatch):
    best, timings, built = _run(tune, monkeypatch, clusters=set(), angle_wrap=1)
    assert best == {"threads_per_cta": 1024, "ctas_per_sm": 1, "sell_window": 1024}
    assert len(timings) == len(built) == 18
    assert all(o["angle_wrap"] == 1 and o["tol"] == 0.0 for o in built)


def test_the_layout_may_decide(tune, monkeypatch):
    best, timings, _ = _run(tune, monkeypatch, clusters={1024},
                            candidates={"threads_per_cta": (256, 512), "sell_window": (32, 1024)})
    assert best == {"sell_window": 1024}
    assert [c for c, _ in timings] == [{"threads_per_cta": 256, "sell_window": 32}, {"sell_window": 1024},
                                       {"threads_per_cta": 512, "sell_window": 32}]
