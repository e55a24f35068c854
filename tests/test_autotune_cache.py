"""The autotuner's cache without a GPU: a choice stored under another work-item rule is not applied."""
import json

from mertens_bound_b200 import autotune


class FakePlan:
    """300 candidates in one group; configuration 4/0/1.0 is the fastest."""

    class table:
        device = 0

    counts, P = [300], 300

    def __init__(self):
        self.applied = None

    def tier_terms(self):
        return 1e6, 9e6

    def group_info(self, g):
        return {"n_T": 60_000}

    def set_schedule(self, s):
        self.sched = s

    def configure(self, *cfg):
        self.applied = cfg

    def time(self, reps):
        return 1.0 if self.applied[0] == 4 else 2.0


def test_choice_of_another_rule_is_not_applied(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("MB_AUTOTUNE_CACHE", str(path))
    space = [(2, 0, 1.0), (4, 0, 1.0)]
    key = "|".join(p for p in autotune.workload_key(FakePlan()).split("|") if not p.startswith("R"))
    stale = {"config": [2, 1, 0.5, 3], "ms": 0.5}
    path.write_text(json.dumps({key: stale, key + "|R1": stale}))
    plan = FakePlan()
    r = autotune.autotune(plan, space=space, schedules=(0,))
    assert not r["cached"] and plan.applied == (4, 0, 1.0)
    again = autotune.autotune(plan, space=space, schedules=(0,))
    assert again["cached"] and plan.applied == (4, 0, 1.0)
    assert json.loads(path.read_text())[key] == stale        # other entries are kept
    monkeypatch.setattr(autotune, "RULE", autotune.RULE + 1)
    assert not autotune.autotune(plan, space=space, schedules=(0,))["cached"]
