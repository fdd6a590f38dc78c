"""With symmetry groups the iteration forms only the bubble rows and FL.K3 blocks that its work items read;
inspection (fdga_get_named) still gives whole arrays.  Against the oracle, 1e-10 of the largest entry (the
plain path's tolerance), with a reference system so that FL does not vanish."""
import numpy as np
import pytest

from helpers import make_gpu, make_oracle

pytestmark = pytest.mark.gpu

NL = dict(kind="hubbard", T=0.4, U=1.5, mu=0.3, t1=1.0, t2=-0.2, mPi_factor=4, refvertex_noise=0.05, seed=7)
CASES = {
    "L4": dict(NL, L=4, nG=8, nK1=8, nK2=(4, 5), nK3=(3, 4)),
    "L3": dict(NL, L=3, nG=7, nK1=6, nK2=(5, 3), nK3=(4, 2)),
    "L5": dict(NL, L=5, nG=6, nK1=5, nK2=(3, 3), nK3=(2, 3)),
    "short_mesh": dict(NL, L=2, nG=8, nK1=6, nK2=(4, 4), nK3=(3, 3), mPi_factor=1),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_inspected_arrays_are_whole(name, precision):
    from fdgasolver.models import hubbard_bare_Green
    cfg = dict(CASES[name])
    cfg["G0"] = hubbard_bare_Green(cfg["T"], cfg["nG"], cfg["L"], mu=0.0, t1=1.0)
    gpu, orc = make_gpu(cfg, True), make_oracle(cfg, True)
    rng = np.random.default_rng(3)
    x = orc.flatten()
    x = x + 0.05 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    gpu.set_precision(precision)
    for _ in range(2):  # a second state: rows left from the first would show
        x = orc.residual(x, "fdPA") + x
        gpu.fixed_point(x, "fdPA")
    orc.residual(x, "fdPA")
    tol = 1e-10 if precision == "fp64" else 1e-5
    for arr in ["Pipp", "Piph"] + [f"FL.{c}.{k}" for c in "pta" for k in ("K2", "K3")]:
        a, b = gpu.get(arr), orc.get(arr)
        assert np.abs(b).max() > 0
        assert np.abs(a - b).max() < tol * np.abs(b).max(), arr
        assert np.array_equal(gpu.get(arr), a)
    gpu.close()
