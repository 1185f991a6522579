"""od_get_state where its copies change (states up to 64 KB, 1365 ions, in one): the set positions and
velocities to the last bit of the device's words, together, alone and one more or fewer ions."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from tests._util import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 255, 1365, 1366, 5461])
def test_state_together_and_alone(gpu_lib, N):
    holder, pos, vel = case(N=N, n=4, seed=N, trap=np.zeros(15))[:3]
    lib = _lib.load()
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        p, v = eng.get_state()
        alone = [np.empty_like(p), np.empty_like(v)]
        _lib.check(lib.od_get_state(eng.h, _lib._dptr(alone[0]), None, N), eng.h)
        _lib.check(lib.od_get_state(eng.h, None, _lib._dptr(alone[1]), N), eng.h)
        eng.set_state(p, v)
        again = eng.get_state()
    assert np.array_equal(p, alone[0]) and np.array_equal(v, alone[1])
    assert np.array_equal(p, again[0]) and np.array_equal(v, again[1])
    # one rounding of a component to FP32: 6e-8 of the cell size (positions), of itself (velocities)
    assert np.abs(p - pos).max() <= 6e-8 * np.abs(pos).max() + 6e-8 * holder.cfg.r_D_e
    assert np.all(np.abs(v - vel) <= 6e-8 * np.abs(vel))


@pytest.mark.parametrize("N", [2, 1365, 1366])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_refused_state_changes_nothing(gpu_lib, N, bad):
    holder, pos, vel = case(N=N, n=4, seed=N, trap=np.zeros(15))[:3]
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        before = eng.get_state()
        for which, at in ((0, 0), (0, -1), (1, 0), (1, -1)):
            x = [pos.copy(), vel.copy()]
            x[which].reshape(-1)[at] = bad
            with pytest.raises(_lib.OpenDustError) as e:
                eng.set_state(*x)
            assert e.value.status == 1
        after = eng.get_state()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
