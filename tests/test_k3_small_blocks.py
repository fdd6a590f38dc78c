"""The FP64 map's K3 contractions of blocks below Nν3 = 32 on warp-level digit products (fdga_k3_mma.cu,
the default there) against the FP64 CUDA-core GEMMs (option k3_fp64_tensor_cores = 0).

Sizes: one to four 8-wide chunks, full and ragged.  Tolerance per flatten block: at most 64 product terms,
each within 2^-54 of (row bound)·(column bound), the bounds within a factor 2 of the largest entries and
the block's largest output at least 1/64 of that product: 64 · 4 · 64 · 2^-54 < 1e-12."""
import numpy as np
import pytest

from helpers import blocks, blockwise_rel_err, make_gpu

pytestmark = pytest.mark.gpu


def _cfg(n, kind):
    base = dict(kind=kind, T=0.3, U=1.5, nG=n + 6, nK1=n + 4, nK2=(4, n + 1), nK3=(3, n), mPi_factor=4)
    if kind == "siam":
        return dict(base, e=0.2, Delta=0.5, D=10.0)
    return dict(base, mu=0.3, t1=1.0, t2=-0.2, L=3, refvertex_noise=0.05, seed=5)


def _state(gpu, rng, strategy="fdPA"):
    x = gpu.flatten()
    x = x + 0.05 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    return gpu.fixed_point(x, strategy) + x


@pytest.mark.parametrize("kind", ["siam", "hubbard"])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 7, 8, 9, 11, 12, 13, 15])
def test_map_and_tangent(n, kind):
    rng = np.random.default_rng(n)
    cfg = _cfg(n, kind)
    G0 = 0.3 * (rng.standard_normal((2 * cfg["nG"], 9 if kind == "hubbard" else 1)) + 0j)
    gpu = make_gpu(dict(cfg, G0=G0.reshape(-1) if kind == "siam" else G0), True)  # Π0 ≠ 0
    for strategy in ("fdPA", "scPA"):
        y = _state(gpu, rng, strategy)
        v = rng.standard_normal(y.size) + 1j * rng.standard_normal(y.size)
        out = []
        for opt in (0, 2):
            gpu.set_option("k3_fp64_tensor_cores", opt)
            f = gpu.fixed_point(y, strategy) + y
            gpu.unflatten(y)
            out.append((f, gpu.frule(v, strategy)[1], gpu.get("FL.p.K3")))
        for a, b in zip(out[0][:2], out[1][:2]):
            assert blockwise_rel_err(cfg, b, a) < 1e-12
        assert not np.array_equal(out[0][0], out[1][0])  # both paths ran
        if strategy == "fdPA" and kind == "hubbard":  # (a bare reference vertex has FL.K3 = 0)
            assert np.abs(out[0][2]).max() > 0
            assert np.abs(out[1][2] - out[0][2]).max() < 1e-12 * np.abs(out[0][2]).max()
    gpu.close()


@pytest.mark.parametrize("n", [4, 11])
def test_nan_reaches_the_same_entries(n):
    cfg = _cfg(n, "siam")
    rng = np.random.default_rng(n)
    gpu = make_gpu(cfg, False)
    y = _state(gpu, rng)
    (_, s, e) = [b for b in blocks(cfg) if b[0] == "a.K3"][0]
    y[(s + e) // 2 + 1] = np.nan
    bad = []
    for opt in (0, 2):
        gpu.set_option("k3_fp64_tensor_cores", opt)
        bad.append(np.isnan(gpu.fixed_point(y, "fdPA")))
    k3 = [(s, e) for name, s, e in blocks(cfg) if name.endswith("K3")]
    assert any(bad[0][s:e].any() for s, e in k3)
    for s, e in k3:
        assert np.array_equal(bad[0][s:e], bad[1][s:e])
    gpu.close()
