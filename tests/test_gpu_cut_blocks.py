"""GPU test of the cutoff kernel over 32-ion blocks (cutoff variant 3) at the sizes where its
lists and units change: one block, one tile, a ragged tail, a snapshot with fewer ions than the
simulation, one and several tiles per unit, both paddings, switching and hard cutoff; and a
lattice on which thousands of pairs lie exactly at the hard cutoff (the exact pass of every
batch). Against the FP64 oracle on the same float positions; tolerance 1e-5 of max(|force|, 1 % of
the rms force) per ion, the FP32 bound of the other cutoff tests with a floor for the lattice's
nearly balanced ions."""
import numpy as np
import pytest

from opendust_gb300 import _lib, workloads
from oracle import oracle
from tests._util import case, rel_err_per_ion

pytestmark = pytest.mark.gpu


def _check(holder, pos, plan, what):
    n = pos.shape[0]
    with _lib.Engine(holder) as eng:
        if plan:
            eng.set_pair_plan(*plan)
        assert eng.pair_plan()["variant"] == 3
        f = eng.force_snapshot(pos)
        f2 = eng.force_snapshot(pos)
    assert np.array_equal(f, f2)
    idx = np.arange(n) if n <= 4096 else np.unique(np.r_[0:100, n - 100:n, np.arange(0, n, max(1, n // 800))])
    ref = oracle.force_targets(holder, pos, idx, round32=True)
    if not np.any(ref):
        assert not np.any(f[idx])
        return
    err = rel_err_per_ion(f[idx], ref, floor_frac=0.01)
    print(f"{what}: per-ion rel err max {err.max():.3e}")
    assert err.max() <= 1e-5


@pytest.mark.parametrize("hard", [False, True])
@pytest.mark.parametrize("N,n,plan", [(2, 2, None), (33, 33, None), (64, 64, None), (65, 65, (256, 4, 3)),
                                      (512, 512, None), (513, 513, (256, 4, 3)), (1500, 700, None),
                                      (5000, 33, None), (131072, 131072, None), (131073, 131073, None),
                                      (200000, 200000, (256, 4, 3))])
def test_block_sizes(gpu_lib, N, n, plan, hard):
    kw = {"switch_distance": 0.0} if hard else {}
    holder, pos, *_ = case(N=N, n=4, seed=31, builder=workloads.field_chain, trap=np.zeros(15), **kw)
    _check(holder, pos[:n], plan, f"N={N} n={n} plan {plan} hard {hard}")


@pytest.mark.parametrize("hard", [False, True])
def test_lattice_pairs_at_the_cutoff(gpu_lib, hard):
    kw = {"switch_distance": 0.0} if hard else {}
    holder, pos, vel, plasma, *_ = case(N=3600, n=4, seed=32, builder=workloads.field_chain,
                                        trap=np.zeros(15), **kw)
    g = np.arange(16) * 0.25 - 1.875  # multiples of 1/8 lambda: pairs exactly 2 lambda apart
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    x = x[np.random.default_rng(4).permutation(len(x))[:3600]]
    _check(holder, x * plasma.r_D_e, None, f"lattice hard {hard}")
