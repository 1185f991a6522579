"""The FP64 tail's series against the oracle: charges, momentum of collected ions, grain-grain forces and
orbit forces of a few steps, with no, one and many ions collected by the grains in the first step. The
charge counts the collected ions: one more or fewer changes it by q_s, and whole numbers of q_s are
compared. FP64 arithmetic on FP32 velocities: 1e-5 of the momentum sums, 1e-9 of charges and grain-grain
forces; 1e-4 of the orbit forces, as the other comparisons of steps."""
import numpy as np
import pytest

from opendust_gb300 import _lib, build_simulation, setup_host, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 3, 16])
@pytest.mark.parametrize("N,hits", [(300, 0), (2048, 1), (5000, 40)])
def test_tail_series(gpu_lib, N, hits, P):
    plasma, sim, _, dist, ext = workloads.small_plain(N=N, n=4)
    lam, r_g = plasma.r_D_e, 1e-5
    grains = [workloads.DustParticle(0.0, 0.0, (k - (P - 1) / 2.0) * 0.3 * lam, r_g, "consistent", -1e-15)
              for k in range(P)]
    holder, _ = build_simulation(plasma, sim, grains, dist, seed=3, trap=np.zeros(15), **ext)
    pos, vel = setup_host.initial_state(N, sim.R, sim.H, [(g.x, g.y, g.z, g.r) for g in grains],
                                        plasma.v_fl, plasma.v_T, dist, 3)
    # ions that a step takes from 0.25 lambda away into their grains, to 0.7 radii from the middle
    rng = np.random.default_rng(4)
    which = rng.permutation(N)[:hits]
    centre = np.array([[q.x, q.y, q.z] for q in grains])[rng.integers(P, size=hits)]
    u, w = (d / np.linalg.norm(d, axis=1)[:, None] for d in rng.normal(size=(2, hits, 3)))
    target = centre + 0.7 * r_g * u
    pos[which] = target + 0.25 * lam * w
    vel[which] = (target - pos[which]) / holder.cfg.d_t
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.step(3)
        s = eng.series(0, 3)
    ref = oracle.run(holder, pos, vel, 0, 3, round32=True)
    assert ref["dN"][0].sum() >= hits
    q_s = abs(plasma.e) * sim.N_s
    assert not np.rint((s["q"] - ref["q"]) / q_s).any()
    assert np.abs(s["q"] - ref["q"]).max() <= 1e-9 * np.abs(ref["q"]).max()
    for name, tol in (("collect", 1e-5), ("dust", 1e-9), ("orbit", 1e-4)):
        scale = np.linalg.norm(ref[name])
        err = np.linalg.norm(s[name] - ref[name]) / scale if scale else np.abs(s[name]).max()
        print(f"N={N} hits={hits} P={P} {name}: rel {err:.2e}")
        assert err <= tol, name
