"""The FP64 map's K3 contractions of blocks above Nν3 = 32 on tcgen05 digit products (fdga_k3_oz.cu, the
default there) against the FP64 CUDA-core GEMMs (option k3_fp64_tensor_cores = 0).

Sizes: last column tiles of 16, 32, 48 and 64 real columns, the edges of the three instantiations (Nν3 up to
64, 96, 128).  Tolerance per flatten block: 2 Nν3 product terms, each within 2^-52 of (row bound)·(column
bound), the bounds within a factor 2 of the largest entries and the block's largest output at least 1/64 of
that product: 2 Nν3 · 4 · 64 · 2^-52."""
import numpy as np
import pytest

from helpers import blocks, blockwise_rel_err, make_gpu

pytestmark = pytest.mark.gpu


def _cfg(n):
    return dict(kind="siam", T=0.3, U=1.5, e=0.2, Delta=0.5, D=10.0, nG=n // 2 + 6, nK1=n // 2 + 4,
                nK2=(4, n // 2 + 1), nK3=(2, n // 2), mPi_factor=4)


def _state(gpu, rng):
    x = gpu.flatten()
    x = x + 0.05 * (rng.standard_normal(x.size) + 1j * rng.standard_normal(x.size))
    return gpu.fixed_point(x) + x


@pytest.mark.parametrize("n", [40, 48, 56, 64, 72, 96, 104, 128])
def test_map_and_tangent(n):
    rng = np.random.default_rng(n)
    cfg = _cfg(n)
    G0 = 0.3 * (rng.standard_normal(2 * cfg["nG"]) + 0j)
    gpu = make_gpu(dict(cfg, G0=G0), True)  # Π0 ≠ 0
    y = _state(gpu, rng)
    for name, s, e in blocks(cfg):  # rows and columns of one block a factor 1e12 apart
        if name.endswith("K3"):
            y[s:e] *= 10.0 ** (12 * rng.random(e - s) - 9)
    v = rng.standard_normal(y.size) + 1j * rng.standard_normal(y.size)
    out = []
    for opt in (0, 2):
        gpu.set_option("k3_fp64_tensor_cores", opt)
        assert gpu.query("k3_fp64_tensor_cores") == (opt != 0)
        f = gpu.fixed_point(y) + y
        gpu.unflatten(y)
        out.append((f, gpu.frule(v)[1]))
    for a, b in zip(*out):
        assert blockwise_rel_err(cfg, b, a) < 2 * n * 256 * 2.0 ** -52
    assert not np.array_equal(out[0][0], out[1][0])  # both paths ran
    gpu.close()


@pytest.mark.parametrize("n", [40, 104])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nan_reaches_the_same_entries(n, bad):
    rng = np.random.default_rng(n)
    cfg = _cfg(n)
    gpu = make_gpu(cfg, False)
    y = _state(gpu, rng)
    (_, s, e) = [b for b in blocks(cfg) if b[0] == "a.K3"][0]
    y[(s + e) // 2 + 1] = bad
    out = []
    for opt in (0, 2):
        gpu.set_option("k3_fp64_tensor_cores", opt)
        out.append(np.isfinite(gpu.fixed_point(y)))
    for name, s, e in blocks(cfg):
        if name.endswith("K3"):
            assert np.array_equal(out[0][s:e], out[1][s:e])
    gpu.close()
