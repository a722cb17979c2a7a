"""The autotuner measures only the knobs that change a launch (few particles have launches of their own)."""
import pytest

from bubbles_gb300 import autotune


class FakeSolver:
    """Records the settings it is timed with; every one of them is a little faster than the last."""

    def __init__(self, n, worklist):
        self.n = n
        self.now = {"block_size": 128, "batch_np": 4, "batch_pd": 4, "batch_pf": 4, "prune": 0,
                    "particles_per_thread": 1, "tile_order": 0, "batch_worklist": worklist}
        self.timed = []

    def tuning(self):
        return dict(self.now)

    def set_tuning(self, **values):
        self.now = dict(values)


class FakeBatch(FakeSolver, autotune.BatchSolver):
    def __del__(self):
        pass


def tuned(monkeypatch, g):
    def timed(solver, *args):
        solver.timed.append(dict(solver.now))
        return 1.0 - 1e-3 * len(solver.timed)
    monkeypatch.setattr(autotune, "time_substeps", timed)
    autotune.tune_launches(g, 1e-3, None, 1, False, [])
    return {k for k in g.timed[0] if len({t[k] for t in g.timed}) > 1}


@pytest.mark.parametrize("n,kind,worklist,want", [
    (77825, FakeSolver, 1, {"block_size", "batch_np", "batch_pd", "batch_pf", "particles_per_thread", "tile_order"}),
    (77824, FakeSolver, 1, {"block_size", "tile_order"}),
    (77824, FakeSolver, 2, {"block_size", "tile_order"}),   # a single scene has no work list
    (1440, FakeSolver, 1, {"block_size", "tile_order"}),
    (77824, FakeBatch, 1, {"block_size", "tile_order", "batch_worklist"}),
    (77824, FakeBatch, 2, {"block_size", "tile_order", "batch_worklist", "batch_pd", "batch_pf"}),
    (77825, FakeBatch, 1, {"block_size", "batch_np", "batch_pd", "batch_pf", "particles_per_thread", "tile_order",
                           "batch_worklist"})])
def test_only_knobs_that_act_are_timed(monkeypatch, n, kind, worklist, want):
    assert tuned(monkeypatch, kind(n, worklist)) == want
