"""CPU test of the persisted plans of single simulations (tuning.tuned_plan): entries of the tuner that
left the default kernel out below 8192 ions are measured again, new ones are reused."""
from opendust_gb300 import tuning


class FakeEngine:
    def __init__(self, n):
        self.n, self.tuned, self.plan = n, 0, None

    def autotune(self, use_cache):
        self.tuned += 1

    def pair_plan(self):
        return dict(threads=256, targets_per_thread=4, variant=7, jsplit=1024)

    def set_pair_plan(self, *plan):
        self.plan = plan


def test_plans_of_the_old_tuner_are_measured_again(tmp_path):
    path = str(tmp_path / "plans.json")
    model = tuning.gpu_model(0)
    old = tuning.PlanCache(path)
    old.put("single", model, 2000, (128, 1, 0, 8))
    old.put("batch", model, 2000, (4, 1024))
    eng = FakeEngine(2000)
    for _ in range(2):
        assert tuning.tuned_plan(eng, cache=tuning.PlanCache(path)) == (256, 4, 7, 1024)
        assert eng.plan == (256, 4, 7, 1024)
    assert eng.tuned == 1
    assert tuning.PlanCache(path).get("batch", model, 2000) == (4, 1024)
