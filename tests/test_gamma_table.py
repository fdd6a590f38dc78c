"""The nonlocal map with the irreducible vertex tabulated once per (Ω, ν, ω) against the oracle.

Boxes at which the table and its readers have edges: K2 boxes with more bosonic than fermionic frequencies
and the reverse, a bubble mesh no wider than the K1 box (mΠν_factor = 1), RefVertex boxes that are the K3
box, larger than the K2 box, and the bare U; with a reference system (Π0 ≠ 0: the left BSEs count).
Tolerance: the plain path's 1e-10 per flatten block (FP64 sums in another order)."""
import numpy as np
import pytest

from helpers import blockwise_rel_err, make_gpu, make_oracle

pytestmark = pytest.mark.gpu

BASE = dict(kind="hubbard", T=0.4, U=1.5, mu=0.3, t1=1.0, t2=-0.2)
CASES = {
    "wide_bosonic": dict(BASE, L=3, nG=7, nK1=8, nK2=(7, 3), nK3=(5, 2), mPi_factor=4, refvertex_noise=0.05, seed=1),
    "wide_fermionic": dict(BASE, L=4, nG=9, nK1=7, nK2=(2, 7), nK3=(2, 6), mPi_factor=3, refvertex_noise=0.05, seed=2),
    "short_mesh": dict(BASE, L=2, nG=8, nK1=5, nK2=(5, 5), nK3=(4, 5), mPi_factor=1, refvertex_noise=0.05, seed=3),
    "large_nR": dict(BASE, L=3, nG=6, nK1=5, nK2=(3, 3), nK3=(2, 2), mPi_factor=4, refvertex_noise=0.05, nR=(4, 6), seed=4),
    "small_nR": dict(BASE, L=5, nG=6, nK1=6, nK2=(4, 5), nK3=(3, 4), mPi_factor=4, refvertex_noise=0.05, nR=(2, 2), seed=5),
    "bare": dict(BASE, L=3, nG=6, nK1=6, nK2=(4, 4), nK3=(1, 1), mPi_factor=4),
}


@pytest.mark.parametrize("sym", [True, False], ids=["groups", "trivial"])
@pytest.mark.parametrize("name", list(CASES))
def test_map_matches_oracle(name, sym):
    from fdgasolver.models import hubbard_bare_Green
    cfg = dict(CASES[name])
    cfg["G0"] = hubbard_bare_Green(cfg["T"], cfg["nG"], cfg["L"], mu=0.0, t1=1.0)
    gpu, orc = make_gpu(cfg, sym), make_oracle(cfg, sym)
    rng = np.random.default_rng(9)
    x = orc.flatten()
    x = x + 0.05 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    for strategy in ("fdPA", "scPA", "fdPA_1loop", "fdPA"):
        y = orc.residual(x, strategy) + x
        assert blockwise_rel_err(cfg, gpu.fixed_point(x, strategy) + x, y) < 1e-10
        x = y
    gpu.close()


@pytest.mark.parametrize("sym", [True, False], ids=["groups", "trivial"])
@pytest.mark.parametrize("name", list(CASES))
def test_adjoint_is_the_transpose_of_the_tangent(name, sym):
    """<ȳ, J v> = <Jᵀ ȳ, v> to 1e-12 of |ȳ| |J v| (both sides are FP64 sums of the same terms)."""
    from fdgasolver.models import hubbard_bare_Green
    cfg = dict(CASES[name])
    cfg["G0"] = hubbard_bare_Green(cfg["T"], cfg["nG"], cfg["L"], mu=0.0, t1=1.0)
    gpu = make_gpu(cfg, sym)
    rng = np.random.default_rng(10)
    noise = lambda: rng.standard_normal(gpu.state_len) + 1j * rng.standard_normal(gpu.state_len)  # noqa: E731
    for strategy in ("fdPA", "scPA"):
        gpu.unflatten(gpu.fixed_point(0.05 * noise(), strategy))
        x = gpu.flatten()
        v, yb = noise(), noise()
        jv = gpu.frule(v, strategy)[1]
        gpu.unflatten(x)
        xb = gpu.rrule(yb, strategy)[1]
        a, b = np.vdot(yb, jv).real, np.vdot(xb, v).real
        assert abs(a - b) < 1e-12 * np.linalg.norm(yb) * np.linalg.norm(jv)
    gpu.close()
