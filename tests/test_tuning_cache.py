"""Plan.autotune's cache file: results of an earlier library, whose candidate numbers meant other
kernels, are not applied, and a stored tuning that the plan rejects is timed again.  The library
call is a stand-in, so the test runs without a GPU."""
import json
from types import SimpleNamespace

import tarang_b200 as tb
from tarang_b200 import _lib as L
from tarang_b200 import solver

TIMED = {"variant": [1, 0, 0, 2, 0], "blocks_per_sm": [0, 0, 0, 0, 0]}


class FakePlan(solver.Plan):
    def __init__(self, rejects=()):
        self.h = None
        self.N, self.basis, self.precision = (64, 64, 64), "FFF", "f32"
        self.cfg = SimpleNamespace(nlin_form=1, dealias_mode=2, force_type=0)
        self.rejects, self.applied, self.timings = list(rejects), None, 0

        def autotune(h, reps, buf, n):
            self.timings += 1
            self.applied = TIMED
            buf.value = json.dumps({"final": TIMED}).encode()
            return 0
        self.lib = SimpleNamespace(ts_plan_autotune=autotune, ts_last_error=lambda: b"")

    def set_tuning(self, tuning):
        if tuning in self.rejects:
            raise tb.TsError(L.TS_ERR_ARG, "ts_plan_set_tuning")
        self.applied = tuning

    def tuning(self):
        return self.applied


def key_before(plan):
    """the key as it was before the candidates were renumbered"""
    c = plan.cfg
    dev = plan.tuning_key().split("|")[0]
    return (f"{dev}|{plan.basis}|{'x'.join(map(str, plan.N))}|{plan.precision}|form{c.nlin_form}"
            f"|dealias{c.dealias_mode}|force{c.force_type}")


def test_results_of_another_candidate_set_are_not_applied(tmp_path):
    plan = FakePlan()
    cache = tmp_path / "tuning.json"
    old = {"variant": [0, 3, 1, 1, 2], "blocks_per_sm": [0, 0, 0, 3, 0]}
    cache.write_text(json.dumps({key_before(plan): old}))
    rep = plan.autotune(cache=str(cache))
    assert plan.timings == 1 and not rep.get("cached") and plan.applied == TIMED
    again = plan.autotune(cache=str(cache))
    assert plan.timings == 1 and again == {"cached": True, "tuning": TIMED}
    assert json.loads(cache.read_text())[key_before(plan)] == old  # the earlier library's entry stays


def test_a_rejected_tuning_is_timed_again(tmp_path):
    gone = {"variant": [0, 0, 4, 0, 0], "blocks_per_sm": [0, 0, 0, 0, 0]}
    plan = FakePlan(rejects=[gone])
    cache = tmp_path / "tuning.json"
    cache.write_text(json.dumps({plan.tuning_key(): gone}))
    rep = plan.autotune(cache=str(cache))
    assert plan.timings == 1 and rep["tuning"] == TIMED
    assert json.loads(cache.read_text())[plan.tuning_key()] == TIMED
