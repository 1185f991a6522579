"""GPU test of the allocation-free entry's source chunks where their rule changes: 64-source chunks
below 2048 padded ions, 128 above, twice the blocks above 76 target tiles (19456 ions), and the
scratch's limit. Against the FP64 oracle on the same float positions; tolerance 1e-5 per ion, the
FP32 bound of the other force tests. Far ions keep the relative accuracy of their small forces, and
a position that is not finite makes every force NaN."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from oracle import oracle
from tests._util import case, rel_err_per_ion
from tests.test_zz_no_alloc import _static_forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 511, 513, 1536, 1537, 2049, 19456, 19457, 32767])
def test_chunk_rule(gpu_lib, n):
    torch = pytest.importorskip("torch")
    holder, pos, _, plasma, sim, _ = case(N=max(n, 2048), n=4, seed=61, trap=np.zeros(15))
    pos = pos[:n]
    got = _static_forces(_lib.load(), pos, plasma, sim, torch)
    idx = np.arange(n) if n <= 4096 else np.unique(np.r_[0:100, n - 100:n, np.arange(0, n, n // 800)])
    err = rel_err_per_ion(got[idx], oracle.force_targets(holder, pos, idx, round32=True))
    print(f"static n={n} vs FP64 oracle: max {err.max():.3e}")
    assert err.max() <= 1e-5


def test_far_ions_and_nan(gpu_lib):
    torch = pytest.importorskip("torch")
    holder, pos, _, plasma, sim, _ = case(N=2048, n=4, seed=62, trap=np.zeros(15))
    lam = plasma.r_D_e
    x = np.array([[0.0, 0.0, -14.0], [0.0, 0.0, 14.0], [0.25, 0.0, 14.0]]) * lam
    got = _static_forces(_lib.load(), x, plasma, sim, torch)
    ref = oracle.force_targets(holder, x, np.arange(3), round32=True)
    assert rel_err_per_ion(got, ref).max() <= 1e-5
    x[2, 0] = np.nan
    assert np.isnan(_static_forces(_lib.load(), x, plasma, sim, torch)).all()
