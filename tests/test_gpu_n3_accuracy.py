"""Accuracy of the default all-pairs forces from 2^14 to 2^15 ions against FP64 sums over the same
positions: the median relative error per ion is no larger than that of the 2 x 2 tile-pair kernel that
was the default there (measured on these sizes, uniform ions in the cylinder, mean of eight seeds)."""
import numpy as np
import pytest
import torch

from opendust_gb300 import _lib
from tests._util import case

pytestmark = pytest.mark.gpu


def forces_fp64(x, rho):
    x = torch.tensor(x, dtype=torch.float64, device="cuda")
    out = torch.empty_like(x)
    rows = 2**25 // x.shape[0]
    for i in range(0, x.shape[0], rows):
        d = x[i:i + rows, None, :] - x[None, :, :]
        r = torch.sqrt((d * d).sum(2))
        r = torch.where(r == 0, torch.full_like(r, torch.inf), r)
        s = 1.0 / (r + rho)
        out[i:i + rows] = ((torch.exp(-r) * s * (1.0 + s) / r)[:, :, None] * d).sum(1)
    return out.cpu().numpy()


@pytest.mark.parametrize("N,bound", [(16385, 5.842e-8), (20011, 5.551e-8), (25000, 5.298e-8),
                                     (32768, 4.961e-8)])
def test_error_from_2_14_to_2_15_ions(gpu_lib, N, bound):
    holder, _, _, plasma, sim, _ = case(N=N, n=4, seed=1, trap=np.zeros(15))
    lam, q_s = plasma.r_D_e, abs(plasma.e) * sim.N_s
    unit = q_s * q_s / (4.0 * np.pi * plasma.eps_0) / lam**2
    med = []
    with _lib.Engine(holder) as eng:
        for seed in range(4):
            rng = np.random.default_rng(seed)
            r, th = 3.0 * np.sqrt(rng.random(N)), 2.0 * np.pi * rng.random(N)
            x = np.stack([r * np.cos(th), r * np.sin(th), 6.0 * (rng.random(N) - 0.5)], 1)
            x = x.astype(np.float32).astype(np.float64)
            ref = unit * forces_fp64(x, holder.cfg.r_0 / lam)
            f = eng.force_snapshot(x * lam)
            med.append(np.median(np.linalg.norm(f - ref, axis=1) / np.linalg.norm(ref, axis=1)))
    print(f"N={N}: median relative error {np.mean(med):.3e}, 2 x 2 tile pairs {bound:.3e}")
    assert np.mean(med) <= bound
