"""GPU test of the cutoff's cell sort where its rules change: the cell grid's sizes (8, 16 and 32
cells per axis), the scan inside the scatter and the one of its own (above 8192 cells), a crowded
cell, and a cell with more ions than the sort takes, which is an error. Against the FP64 oracle on the same float positions; tolerance 1e-5 of max(|force|, 1 % of the
rms force) per ion, the FP32 bound of the other cutoff tests."""
import numpy as np
import pytest

from opendust_gb300 import _lib, workloads
from oracle import oracle
from tests._util import case, rel_err_per_ion

pytestmark = pytest.mark.gpu


def _check(eng, holder, pos):
    n = pos.shape[0]
    f = eng.force_snapshot(pos)
    assert np.array_equal(f, eng.force_snapshot(pos))
    idx = np.arange(n) if n <= 4096 else np.unique(np.r_[0:100, n - 100:n, np.arange(0, n, max(1, n // 600))])
    err = rel_err_per_ion(f[idx], oracle.force_targets(holder, pos, idx, round32=True), floor_frac=0.01)
    print(f"n={n}: per-ion rel err max {err.max():.3e}")
    assert err.max() <= 1e-5


@pytest.mark.parametrize("N", [5792, 5793, 46340, 46342])
def test_cell_grids(gpu_lib, N):
    holder, pos, *_ = case(N=N, n=4, seed=71, builder=workloads.field_chain, trap=np.zeros(15))
    with _lib.Engine(holder) as eng:
        assert eng.pair_plan()["variant"] == 3
        _check(eng, holder, pos)
        _check(eng, holder, pos[:N // 3])


def test_crowded_cell(gpu_lib):
    holder, pos, _, plasma, *_ = case(N=9000, n=4, seed=72, builder=workloads.field_chain, trap=np.zeros(15))
    rng = np.random.default_rng(3)
    clump = pos.copy()
    clump[2000:3900] = plasma.r_D_e * (np.array([1.0, 1.0, 1.0]) + 0.05 * rng.random((1900, 3)))
    full = pos.copy()
    full[2000:4200] = plasma.r_D_e * (np.array([1.0, 1.0, 1.0]) + 0.05 * rng.random((2200, 3)))
    with _lib.Engine(holder) as eng:
        _check(eng, holder, clump)
        with pytest.raises(_lib.OpenDustError):
            eng.force_snapshot(full)
