"""GPU test of the each-pair-once kernel's work split (variant 7): ion counts on both sides of
every change of the split (group pairs in 4, 2 and 1 parts; 4 x 4 and 8 x 2 ions per lane), the
smallest sizes, and slices longer than a row, against the FP64 oracle. Tolerance: per-ion
relative error 1e-5, the bound of the other force tests."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from oracle import oracle
from tests._util import case, plant_close_pairs, rel_err_per_ion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,plan", [(130, None), (512, None), (513, None), (4096, None), (4097, None),
                                    (12288, None), (12289, None), (65536, None), (65537, None),
                                    (4097, (256, 2, 7, 4096)), (700, (256, 8, 7, 4096)),
                                    (20000, (256, 8, 7, 4096)), (20000, (256, 2, 7, 512))])
def test_split_boundaries(gpu_lib, N, plan):
    holder, pos, vel, plasma, sim, grains = case(N=max(N, 400), n=4, seed=23)
    pos = pos[:N]
    if N > 300:
        pos = plant_close_pairs(pos, plasma.r_D_e, np.random.default_rng(3), n_pairs=32, dmin=2e-4)
    with _lib.Engine(holder) as eng:
        if plan:
            eng.set_pair_plan(*plan)
        assert eng.pair_plan()["variant"] == 7
        f = eng.force_snapshot(pos)
        f2 = eng.force_snapshot(pos)
    assert np.array_equal(f, f2)
    idx = np.arange(N) if N <= 4097 else np.unique(np.r_[0:200, N - 200:N, np.arange(0, N, max(1, N // 1500))])
    err = rel_err_per_ion(f[idx], oracle.force_targets(holder, pos, idx, round32=True))
    print(f"N={N} plan {plan}: per-ion rel err max {err.max():.3e}")
    assert err.max() <= 1e-5


@pytest.mark.parametrize("N", [7680, 7681, 15872, 15873])
def test_part_boundaries(gpu_lib, N):
    """group pairs in 4 parts up to 7680 padded ions, in 2 below 2^14"""
    test_split_boundaries(gpu_lib, N, None)
