"""The cutoff's cell scan in one block: a domain so tall that its column of cubes has more cells than the
scatter scans itself (8192) and no multiple of 4096. Against the FP64 oracle; tolerance 1e-5 of
max(|force|, 1 % of the rms force) per ion, the FP32 bound of the other cutoff tests."""
import numpy as np
import pytest

import opendust_gb300 as od
from opendust_gb300 import _lib, workloads
from oracle import oracle
from tests._util import rel_err_per_ion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tall", [17, 23])  # cubes of 8^3 cells: 8704 and 11776
def test_one_block_scan(gpu_lib, tall):
    plasma = od.PlasmaParametersInSIUnitsMaxwell(workloads.T_I, workloads.T_E, workloads.N_INF, 1.0,
                                                 workloads.M_AR)
    lam, N = plasma.r_D_e, 6001
    sim = od.SimulationParametersInSIUnits(1.0 * lam, 2.0 * tall * lam, N, 4, 1e-10, plasma)
    grains = [od.DustParticle(0.0, 0.0, 0.0, 5e-6, "consistent", -1e-15)]
    holder, _ = od.build_simulation(plasma, sim, grains, "Maxwellian", seed=1, trap=np.zeros(15),
                                    cutoff_distance=2.0 * lam, switch_distance=1.875 * lam)
    rng = np.random.default_rng(tall)
    with _lib.Engine(holder) as eng:
        assert eng.pair_plan()["variant"] == 3
        for n in (N, 1000):
            r, th = np.sqrt(rng.random(n)), 2.0 * np.pi * rng.random(n)
            x = np.stack([r * np.cos(th), r * np.sin(th), 2.0 * tall * (rng.random(n) - 0.5)], 1)
            pos = lam * x.astype(np.float32).astype(np.float64)
            f = eng.force_snapshot(pos)
            assert np.array_equal(f, eng.force_snapshot(pos))
            ref = oracle.force_targets(holder, pos, np.arange(n), round32=True)
            err = rel_err_per_ion(f, ref, floor_frac=0.01)
            print(f"{tall} cubes, n={n}: per-ion rel err max {err.max():.3e}")
            assert err.max() <= 1e-5
