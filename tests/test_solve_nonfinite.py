"""Solvers on states that are or become NaN: they report FDGA_ERR_NONFINITE, never convergence.

Free electrons (U = 0) with Gbare(ν) = sign ν and Σ(ν) = -2 sign ν: the first image is finite, the plain step
of weight 1/2 lands on 1/Gbare + Σ = 0, and the second image is NaN wherever it is not 0.  With symmetry groups
the solver's vectors hold one value per key from the first image on, so the NaN appears on that path."""
import numpy as np
import pytest

from helpers import make_gpu

pytestmark = pytest.mark.gpu

LOCAL = dict(kind="siam", T=0.1, U=1.0, e=0.2, Delta=0.5, D=10.0, nG=16, nK1=16, nK2=(5, 4), nK3=(4, 4), mPi_factor=6)
NL = dict(kind="hubbard", T=0.4, U=1.5, mu=0.1, t1=1.0, L=3, nG=6, nK1=6, nK2=(3, 2), nK3=(2, 2), mPi_factor=3,
          refvertex_noise=0.05, seed=3)
NONFINITE = 5


def _rc(call):
    from fdgasolver._lib import FdgaError
    with pytest.raises(FdgaError) as e:
        call()
    return e.value.code


@pytest.mark.parametrize("sym", [True, False], ids=["groups", "trivial"])
@pytest.mark.parametrize("L", [0, 2])
@pytest.mark.parametrize("mem", [0, 8])
def test_nan_after_the_first_step(sym, L, mem):
    import fdgasolver as F
    nG = 6
    sg = np.sign(np.arange(-nG, nG) + 0.5)[:, None] * np.ones((1, max(1, L) ** 2))
    args, rv = (6, (3, 3), (2, 2)), F.RefVertex(0.2, 0.0)
    if L:
        S = F.NL_ParquetSolver(*args, L, sg + 0j, 0j * sg, 0j * sg, rv, mPi_factor=4)
    else:
        S = F.ParquetSolver(*args, sg + 0j, 0j * sg, 0j * sg, rv, mPi_factor=4)
    if sym:
        S.init_sym_grp()
    x = np.zeros(S.state_len, dtype=complex)
    x[-sg.size:] = -2 * sg.T.reshape(-1)
    S.unflatten(x)
    r = S.solve(maxiter=1, tol=1e-4, delta=0.5, mem=mem)
    assert r["residual"] == 2.0 and not r["converged"]
    S.unflatten(x)
    assert _rc(lambda: S.solve(maxiter=5, tol=1e-4, delta=0.5, mem=mem)) == NONFINITE
    S.close()


@pytest.mark.parametrize("sym", [True, False], ids=["groups", "trivial"])
@pytest.mark.parametrize("cfg", [LOCAL, NL], ids=["local", "nonlocal"])
@pytest.mark.parametrize("solver", ["solve", "solve_mixed", "solve_newton"])
def test_nan_in_the_start(sym, cfg, solver):
    S = make_gpu(cfg, sym)
    every = np.full(S.state_len, np.nan + 0j)
    one = np.zeros(S.state_len, dtype=complex)
    one[S.state_len // 2] = np.nan
    for x in (every, one):
        S.unflatten(x)
        assert _rc(lambda: getattr(S, solver)(maxiter=4, tol=1e-4)) == NONFINITE
    S.close()
