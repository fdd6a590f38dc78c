"""The device Anderson solve on one value per (class, conjugation) key against the oracle's full vectors.

With symmetry groups and a class-symmetric start the solver's vectors hold one value per key; from an
asymmetric start, and without groups, they are full.  All three must follow the oracle's trajectory.
Tolerance: the trajectories differ by the order of the sums, 1e-16 amplified by the condition of the
least-squares history (below 1e6 for at most 8 columns here), so 1e-9 relative."""
import numpy as np
import pytest

from helpers import blockwise_rel_err, make_gpu, make_oracle

LOCAL = dict(kind="siam", T=0.1, U=1.0, e=0.2, Delta=0.5, D=10.0, nG=16, nK1=16, nK2=(5, 4), nK3=(4, 4), mPi_factor=6)
NL = dict(kind="hubbard", T=0.5, U=2.0, mu=0.3, t1=1.0, t2=-0.2, L=4, nG=8, nK1=8, nK2=(3, 3), nK3=(2, 3), mPi_factor=4,
          refvertex_noise=0.05, seed=7)
ODD = dict(kind="hubbard", T=0.4, U=1.5, mu=0.1, t1=1.0, L=3, nG=6, nK1=6, nK2=(3, 2), nK3=(2, 2), mPi_factor=3,
           refvertex_noise=0.05, seed=3)


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [LOCAL, NL, ODD], ids=["local", "nl4", "nl3"])
@pytest.mark.parametrize("mem", [0, 1, 2, 8])
@pytest.mark.parametrize("start", ["groups", "groups_asymmetric", "trivial"])
def test_solve_follows_oracle(cfg, mem, start):
    gpu, orc = make_gpu(cfg, start != "trivial"), make_oracle(cfg, start != "trivial")
    x = gpu.flatten()
    if start == "groups_asymmetric":
        rng = np.random.default_rng(5)
        x = x + 0.01 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    gpu.unflatten(x)
    orc.unflatten(x)
    r = gpu.solve("fdPA", maxiter=11, tol=0.0, delta=0.5, mem=mem)
    o = orc.solve("fdPA", maxiter=11, tol=0.0, beta=0.5, mem=mem)
    assert r["iterations"] == o["iterations"] == 11 and not r["converged"]
    assert np.allclose(r["trace"], o["trace"], rtol=1e-8, atol=1e-10 * o["trace"][0])
    assert blockwise_rel_err(cfg, gpu.flatten(), orc.flatten()) < 1e-9
