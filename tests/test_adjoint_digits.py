"""The adjoint K3 products: on the warp-level digit kernel (k_adj_mma, the default up to Nν3 = 32), and the
launchers' statuses."""
import glob
import os
import re

import numpy as np
import pytest

from helpers import blockwise_rel_err, make_gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fddgasolver.jl_gb300", "csrc")


def test_no_launcher_status_is_dropped():
    """A launcher takes the launch's error out of the runtime (cudaGetLastError), so a call whose status is dropped
    hides a kernel that did not run: none stands as a statement of its own."""
    dropped = []
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for i, line in enumerate(open(f, encoding="utf-8"), 1):
            if re.match(r"\s*((else )?if \(.*\) |else )?launch_\w+(<[^;(]*>)?\(.*;", line):
                dropped.append(f"{os.path.basename(f)}:{i}: {line.strip()}")
    assert not dropped


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7, 11, 12, 15, 16])
@pytest.mark.parametrize("kind", ["siam", "hubbard"])
def test_adjoint_products(n, kind):
    """rrule on the digit products against the CUDA-core GEMMs, two to four 8-wide chunks, full and ragged.
    Tolerance per flatten block: the sums of the adjoint differ by their rounding (1e-16 of at most 1e3 terms)."""
    rng = np.random.default_rng(n)
    cfg = dict(kind=kind, T=0.3, U=1.5, nG=n + 6, nK1=n + 4, nK2=(4, n + 1), nK3=(3, n), mPi_factor=4)
    cfg.update(dict(e=0.2, Delta=0.5, D=10.0) if kind == "siam" else
               dict(mu=0.3, t1=1.0, t2=-0.2, L=2, refvertex_noise=0.05, seed=5))
    G0 = 0.3 * (rng.standard_normal((2 * cfg["nG"], 4 if kind == "hubbard" else 1)) + 0j)
    S = make_gpu(dict(cfg, G0=G0.reshape(-1) if kind == "siam" else G0), True)
    noise = lambda: rng.standard_normal(S.state_len) + 1j * rng.standard_normal(S.state_len)  # noqa: E731
    x = S.fixed_point(0.05 * noise())
    yb = noise()
    out = []
    for opt in (0, 2):
        S.set_option("k3_fp64_tensor_cores", opt)
        S.unflatten(x)
        out.append(S.rrule(yb)[1])
    assert blockwise_rel_err(cfg, out[1], out[0]) < 1e-12
    assert not np.array_equal(out[0], out[1])
    S.close()
