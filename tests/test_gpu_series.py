"""Reads of the result series at the lengths where their copies change (256 KB of rows in one copy,
longer ones split on the device, 16 MB at a time): the same numbers as row by row, whole or in part,
every array or one."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from tests._util import case

pytestmark = pytest.mark.gpu

NAMES = ("q", "orbit", "collect", "dust", "field")


def engine(rows, P):
    holder, pos, vel, plasma, sim, grains = case(N=256, n=rows, seed=P, trap=np.zeros(15),
                                                 builder=_builder(P))
    eng = _lib.Engine(holder)
    eng.set_state(pos, vel)
    eng.step(rows)
    return eng


def _builder(P):
    from opendust_gb300 import workloads

    def build(N, n):
        plasma, sim, grains, dist, ext = workloads.small_plain(N=N, n=n)
        lam = plasma.r_D_e
        grains = [workloads.DustParticle(0.0, 0.0, (k - (P - 1) / 2.0) * 0.3 * lam, 1e-5, "consistent", -1e-15)
                  for k in range(P)]
        return plasma, sim, grains, dist, ext

    return build


@pytest.mark.parametrize("rows,P", [(2520, 1), (2521, 1), (700, 5), (10100, 16)])
def test_long_reads_equal_short_ones(gpu_lib, rows, P):
    with engine(rows, P) as eng:
        whole = eng.series(0, rows)
        step = max(1, (256 << 10) // (104 * P))
        parts = [eng.series(k, min(step, rows - k)) for k in range(0, rows, step)]
        part = eng.series(3, rows - 5)
        for m, name in enumerate(NAMES):
            ref = np.concatenate([p[name] for p in parts])
            assert np.array_equal(whole[name], ref)
            assert np.array_equal(part[name], ref[3:rows - 2])
            one = np.empty_like(ref)
            ptr = [_lib._dptr(one) if k == m else None for k in range(5)]
            _lib.check(_lib.load().od_get_series(eng.h, 0, rows, *ptr), eng.h)
            assert np.array_equal(one, ref)
        assert len(np.unique(whole["q"][:, 0])) > 1 and np.abs(whole["orbit"]).min() > 0
