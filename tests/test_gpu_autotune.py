"""The autotuner against the default plan: the plan it takes steps at most a tenth slower, from the
smallest systems on, and the forces are those of the present state afterwards."""
import time

import numpy as np
import pytest

from opendust_gb300 import _lib
from tests._util import case

pytestmark = pytest.mark.gpu


def step_us(eng, steps=100, tries=7):
    t = []
    for _ in range(tries):
        eng.begin_window()
        t0 = time.perf_counter()
        eng.step(steps)
        t.append(time.perf_counter() - t0)
    return 1e6 * min(t) / steps


@pytest.mark.parametrize("N", [600, 2000, 4000, 7000, 12000])
def test_tuned_plan_is_not_slower_than_the_default(gpu_lib, N):
    holder, pos, vel = case(N=N, n=100, seed=2, trap=np.zeros(15))[:3]
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        before = step_us(eng)
        eng.autotune(use_cache=False)
        tuned = step_us(eng)
        print(f"N={N}: default {before:.1f} us per step, tuned {tuned:.1f} ({eng.pair_plan()})")
        assert tuned <= 1.1 * before
    # a step from the set state: the tuner leaves the sums of that state, not its own launches'. Bounds:
    # forces 1e-5 relative, a step's kick below 1e-2 lambda
    with _lib.Engine(holder) as a, _lib.Engine(holder) as b:
        a.set_state(pos, vel)
        a.autotune(use_cache=False)
        b.set_state(pos, vel)
        a.step(2)
        b.step(2)
        d = np.abs(a.get_state()[0] - b.get_state()[0]).max() / (holder.cfg.r_D_e)
        assert d < 1e-6, d
