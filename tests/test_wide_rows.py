"""Frequency boxes so wide that a row's tables pass the default shared-memory limit (48 KB) of a launch, and K2
boxes so large that a table of the irreducible vertex would dwarf the state.

Tolerance against the oracle: the plain path's 1e-10 per flatten block (FP64 sums in another order); rrule against
frule: 1e-12 of |ȳ| |J v|, as for small boxes."""
import numpy as np
import pytest

from helpers import blockwise_rel_err, make_gpu, make_oracle

pytestmark = pytest.mark.gpu

SIAM = dict(kind="siam", T=0.3, U=1.5, e=0.2, Delta=0.5, D=10.0, nG=8, nK3=(1, 2), mPi_factor=1)
HUB = dict(kind="hubbard", T=0.3, U=1.5, mu=0.3, t1=1.0, t2=-0.2, L=2, nG=8, nK3=(1, 2), mPi_factor=1,
           refvertex_noise=0.05, seed=3)


def _start(S, seed):
    rng = np.random.default_rng(seed)
    return 0.05 * (rng.standard_normal(S.state_len) + 1j * rng.standard_normal(S.state_len))


def _matches_oracle(cfg, sym=True):
    S, orc = make_gpu(cfg, sym), make_oracle(cfg, sym)
    x = _start(S, 1)
    y = orc.residual(x, "fdPA") + x
    err = blockwise_rel_err(cfg, S.fixed_point(x) + x, y)
    S.close()
    assert err < 1e-10


def _transposed(cfg, sym=True):
    S = make_gpu(cfg, sym)
    x = S.fixed_point(_start(S, 2))
    v, yb = _start(S, 3), _start(S, 4)
    S.unflatten(x)
    jv = S.frule(v)[1]
    S.unflatten(x)
    xb = S.rrule(yb)[1]
    S.close()
    assert abs(np.vdot(yb, jv).real - np.vdot(xb, v).real) < 1e-12 * np.linalg.norm(yb) * np.linalg.norm(jv)


def test_each_form_of_k2_raises_its_own_limit():
    """The forms of one kernel (evaluated, tabulated, with a Vertex-valued F0, tangent) have limits of their own:
    rows past 48 KB run in each of them, whichever came first and however wide that was."""
    import fdgasolver as F
    wide, less = dict(nK1=1660, nK2=(1, 4)), dict(nK1=1600, nK2=(1, 4))
    _matches_oracle(dict(SIAM, **wide))  # evaluated: 53 KB
    _matches_oracle(dict(HUB, **less))   # tabulated: 51 KB
    cfg = dict(SIAM, **less)             # Vertex-valued F0 without channels: the map around its RefVertex
    plain = make_gpu(cfg, True)
    Gb = F.siam_bare_Green(cfg["T"], cfg["nG"], Delta=cfg["Delta"], e=cfg["e"], D=cfg["D"])
    F0 = F.Vertex(F.RefVertex(cfg["T"], cfg["U"]), 1, (1, 1), (1, 1), np.zeros(3 * (1 + 2 + 4), dtype=complex))
    S = F.ParquetSolver(cfg["nK1"], cfg["nK2"], cfg["nK3"], Gb, 0 * Gb, 0 * Gb, F0, mPi_factor=1)
    S.init_sym_grp()
    x = _start(S, 5)
    a, b = plain.fixed_point(x) + x, S.fixed_point(x) + x
    assert blockwise_rel_err(cfg, b, a) < 1e-10
    plain.close()
    S.close()


def test_a_tangent_leaves_the_map_its_limit():
    """K2 and SDE rows: a tangent (twice the tables) before a wider plain map."""
    S = make_gpu(dict(SIAM, nK1=1540, nK2=(1, 1540)), True)
    x = S.fixed_point(_start(S, 6))
    S.unflatten(x)
    S.frule(_start(S, 7))
    S.close()
    _matches_oracle(dict(SIAM, nK1=1700, nK2=(1, 1700)))


def test_a_narrower_k3_box_leaves_a_wider_one_its_limit():
    """K3 contractions at Nν3 = 96 after a handle with Nν3 = 72 was prepared: they share kernels."""
    cfg = lambda n: dict(SIAM, nG=n + 4, nK1=n + 2, nK2=(3, n), nK3=(2, n), mPi_factor=2)  # noqa: E731
    S = make_gpu(cfg(48), True)
    x = _start(S, 9)
    make_gpu(cfg(36), True).close()
    y = S.fixed_point(x) + x
    S.unflatten(x)
    S.frule(x)
    S.set_option("k3_fp64_tensor_cores", 0)
    ref = S.fixed_point(x) + x
    S.close()
    assert blockwise_rel_err(cfg(48), y, ref) < 1e-12  # as test_k3_fp64_tensor_cores.py


def test_adjoint_of_wide_fermionic_rows():
    """K2 rows of up to 2 nK2ν = 2560 items: past the 2458 whose values fit 48 KB (nonlocal, trivial groups)."""
    _transposed(dict(HUB, nK1=1280, nK2=(1, 1280)), sym=False)


def test_large_k2_box_fits():
    """nK2 = (170, 170) on 2 x 2: the K2 arrays take 22 MB, a table of the irreducible vertex 5.7 GB."""
    import torch
    cfg = dict(HUB, nK1=170, nK2=(170, 170), nK3=(2, 2), mPi_factor=2)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    S = make_gpu(cfg, True)
    x = S.fixed_point(_start(S, 8))
    S.unflatten(x)
    S.rrule(x)
    S.unflatten(x)
    S.frule(x)
    used = free - torch.cuda.mem_get_info()[0]
    S.close()
    assert used < 2 << 30
    _matches_oracle(cfg)
    _transposed(cfg)
