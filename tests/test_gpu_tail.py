"""GPU test of the step's last kernels at the sizes where their split changes: orbit sums of one
256-ion block, of a ragged last block, of one block per thread block (up to 304 blocks, 77824 ions)
and four; no re-injected ion, some, and more than the blocks that recompute their sums (32 to 304),
with several in one 256-ion block. Two steps against the FP64 oracle: the second starts from the
corrected forces and the updated charges. Bounds: those of the other two-step comparisons, 1e-4
relative (as one norm) for the orbit forces and 1e-5 lambda for the positions, whole numbers equal."""
import numpy as np
import pytest

from opendust_gb300 import _lib, workloads
from oracle import oracle
from tests._util import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("builder", [workloads.small_plain, workloads.field_chain])
@pytest.mark.parametrize("N,leaving", [(256, 0), (257, 1), (2048, 700), (2300, 2300), (77824, 500),
                                       (77825, 500)])
def test_orbit_sums_and_corrections(gpu_lib, builder, N, leaving):
    if N > 4096 and builder is workloads.small_plain:
        pytest.skip("all pairs: the oracle takes minutes")
    holder, pos, vel, plasma, sim, grains = case(N=N, n=4, seed=51, builder=builder, trap=np.zeros(15))
    lam = plasma.r_D_e
    out = np.random.default_rng(5).permutation(N)[:leaving]
    vel[out, :2] = 0.0
    vel[out, 2] = 2.0 * sim.H / holder.cfg.d_t  # through the top face in the first step
    with _lib.Engine(holder) as eng:
        eng.set_state(pos, vel)
        eng.step(2)
        s = eng.series(0, 2)
        p, _ = eng.get_state()
    ref = oracle.run(holder, pos, vel, 0, 2, round32=True)
    if builder is workloads.small_plain:  # the field-driven ions' collisions come before the drift
        assert ref["n_inj"][0] >= leaving
    do = np.linalg.norm(s["orbit"] - ref["orbit"]) / np.linalg.norm(ref["orbit"])
    dpos = np.max(np.abs(p - ref["pos"])) / lam
    print(f"{builder.__name__} N={N}, {ref['n_inj']} re-injected: orbit rel {do:.2e}, max |dx| {dpos:.2e} lambda")
    assert do < 1e-4
    assert dpos < 1e-5
