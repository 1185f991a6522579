"""GPU test of the trap-fit potential grid where its split changes: one point, quads that are not
full, one chunk and several, a chunk across point tiles, one node block and several. Against the
FP64 oracle. Bound 2e-5 relative: a coordinate within 6 lambda is rounded by up to 3e-7, which is
6e-6 of the distance of a point 0.05 lambda from a node; the FP32 terms add about 1e-6."""
import numpy as np
import pytest

from opendust_gb300 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,H", [(0.5, 1.0), (2.6, 5.0), (3.0, 12.0)])
@pytest.mark.parametrize("n", [1, 3, 255, 257, 2049, 20001, 700001])
def test_trap_grid(gpu_lib, R, H, n):
    n_r, n_h = int(R * 10), int(H * 5)
    pot = _lib.trap_potential(R, H, n_r, n_h, n, 11)
    ref = oracle.trap_potential(R, H, n_r, n_h, n, 11)
    err = np.max(np.abs(pot - ref) / np.abs(ref))
    print(f"R={R} H={H}, {n} points: max rel {err:.2e}")
    assert err <= 2e-5
