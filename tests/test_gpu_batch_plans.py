"""Batch members whose all-pairs plan is set through their own handle (od_batch_member): the batch steps
them with that plan. Each-pair-once plans give bitwise the results of the simulation stepped alone with
the same plans; small, ragged and larger members, beside one that keeps its plan."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from tests._util import case

pytestmark = pytest.mark.gpu

ONCE = [(256, 2, 7, 512), (256, 2, 7, 4096), (256, 4, 7, 4096), (256, 8, 7, 2048), (256, 8, 7, 4096)]


def stepped_alone(holder, pos, vel, plan, before, steps):
    with _lib.Engine(holder) as eng:
        eng.set_pair_plan(*_lib.batch_pair_plan(eng.n))
        eng.set_state(pos, vel)
        eng.step(before)
        if plan:
            eng.set_pair_plan(*plan)
        eng.step(steps)
        return (*eng.get_state(), eng.series(0, before + steps))


def stepped_in_batch(members, before, steps):
    """members: (holder, pos, vel, plan or None)"""
    with _lib.Batch() as b:
        slots = [b.add(*m[:3]) for m in members]
        if before:
            b.step(before)
        for s, (*_, plan) in zip(slots, members):
            if plan:
                b.member(s).set_pair_plan(*plan)
        b.step(steps)
        return [(*b.member(s).get_state(), b.member(s).series(0, before + steps)) for s in slots]


def same(a, b):
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert all(np.array_equal(a[2][k], b[2][k]) for k in a[2])


@pytest.mark.parametrize("plan", ONCE)
@pytest.mark.parametrize("N", [300, 9001, 66000])
def test_plan_set_before_the_first_step(gpu_lib, plan, N):
    a = case(N=N, n=8, seed=N, trap=np.zeros(15))[:3]
    c = case(N=2048, n=8, seed=7, trap=np.zeros(15))[:3]
    got = stepped_in_batch([(*a, plan), (*c, None)], 0, 3)
    same(got[0], stepped_alone(*a, plan, 0, 3))
    same(got[1], stepped_alone(*c, None, 0, 3))


@pytest.mark.parametrize("plan", [(256, 1, 5, 0), (128, 1, 5, 7), (256, 2, 2, 0), (256, 1, 0, 0)])
@pytest.mark.parametrize("N", [700, 5000, 20000])
def test_directed_plan_set_before_the_first_step(gpu_lib, plan, N):
    # the batch's directed kernel sums other chains than the handle alone: FP32 rounding apart. The
    # forces of the two agree to 1e-5 (the bound of every all-pairs plan) and a step's kick moves an
    # ion by less than 1e-2 lambda, so the positions agree to 4e-7 lambda after four steps, and to 1e-6
    # with the rounding of the position words (2.4e-7 at 3 lambda)
    a = case(N=N, n=8, seed=N, trap=np.zeros(15))
    plasma = a[3]
    with _lib.Batch() as b:
        s = b.add(*a[:3])
        m = b.member(s)
        m.set_pair_plan(*plan)
        b.step(3)
        p, _ = m.get_state()
        m.step(1)  # alone, with the same slabs
        p4, _ = m.get_state()
    ref = stepped_alone(*a[:3], plan, 0, 3)
    ref4 = stepped_alone(*a[:3], plan, 0, 4)
    d, d4 = (np.abs(x - y[0]).max() / plasma.r_D_e for x, y in ((p, ref), (p4, ref4)))
    print(f"N={N} plan {plan}: {d:.2e} {d4:.2e} lambda")
    assert d < 1e-6 and d4 < 1e-6


@pytest.mark.parametrize("plan", ONCE)
@pytest.mark.parametrize("N", [300, 9001])
def test_plan_changed_between_steps(gpu_lib, plan, N):
    a = case(N=N, n=8, seed=N, trap=np.zeros(15))[:3]
    c = case(N=2048, n=8, seed=7, trap=np.zeros(15))[:3]
    got = stepped_in_batch([(*a, plan), (*c, None)], 2, 4)
    same(got[0], stepped_alone(*a, plan, 2, 4))
    same(got[1], stepped_alone(*c, None, 2, 4))


def test_directed_plan_between_steps_and_back(gpu_lib):
    # bounds as above
    a = case(N=5000, n=8, seed=3, trap=np.zeros(15))
    plans = [(256, 8, 7, 2048), (256, 1, 5, 0), (256, 4, 7, 1024)]
    with _lib.Batch() as b:
        m = b.member(b.add(*a[:3]))
        b.step(1)
        for plan in plans:
            m.set_pair_plan(*plan)
            b.step(1)
        p, _ = m.get_state()
    with _lib.Engine(a[0]) as eng:
        eng.set_pair_plan(*_lib.batch_pair_plan(5000))
        eng.set_state(*a[1:3])
        eng.step(1)
        for plan in plans:
            eng.set_pair_plan(*plan)
            eng.step(1)
        ref, _ = eng.get_state()
    assert np.abs(p - ref).max() / a[3].r_D_e < 1e-6


def test_autotuned_member(gpu_lib):
    # whatever plan the tuner takes, the batch steps the member with it (bounds as above)
    a = case(N=3000, n=8, seed=4, trap=np.zeros(15))
    with _lib.Batch() as b:
        m = b.member(b.add(*a[:3]))
        b.step(2)
        m.autotune(use_cache=False)
        b.step(2)
        p, _ = m.get_state()
    ref = stepped_alone(*a[:3], None, 0, 4)
    assert np.abs(p - ref[0]).max() / a[3].r_D_e < 1e-6
