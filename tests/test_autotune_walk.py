"""Launch shapes the autotuner times: none twice under another name, and choices of
earlier kernels left alone."""
import json

from ghostlight_gb300 import autotune as A


def test_candidates_differ():
    pairs, legs = A.ghost_candidates(False), A.ghost_candidates(True)
    assert pairs == A.GHOST_CANDIDATES
    assert set(legs) <= set(pairs) and len([c for c in legs if c[0] == 0]) == len({c[:2] for c in pairs if c[0] == 0})
    assert [c for c in legs if c[0] > 0] == [c for c in pairs if c[0] > 0]


class _Plan:
    n_items, rays, width, height = 10, 1000, 4, 4

    def __init__(self, walk_tasks):
        self.walk_tasks, self.shape, self.tried = walk_tasks, None, []

    def set_launch(self, *shape):
        self.shape = shape

    def execute(self, *outs, stream=None):
        self.tried.append(self.shape)


def test_choices_of_earlier_kernels_are_not_taken(tmp_path, monkeypatch):
    monkeypatch.setattr(A, "_device_name", lambda: "dev")
    path = tmp_path / "tune.json"
    path.write_text(json.dumps({"ghost|dev|10|1000|16": [1, 0, 4]}))

    class T(A.Tuner):
        def _cuda_timer(self, stream):
            def time_one(run, c):
                run(c)
                return 1.0 if c[0] == 0 else 3.0
            return time_one

    t = T(cache_path=str(path))
    plan = _Plan(7)
    assert A.tune_ghost_plan(plan, (), tuner=t)[0] == 0 and plan.shape[0] == 0
    assert len(set(plan.tried)) == len({c[:2] if c[0] == 0 else c for c in plan.tried})
    # pair by pair is a key of its own
    before = len(plan.tried)
    other = _Plan(0)
    A.tune_ghost_plan(other, (), tuner=t)
    assert set(other.tried) == set(A.GHOST_CANDIDATES) and len(plan.tried) == before
