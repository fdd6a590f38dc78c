"""flatten! / unflatten! on the device (tiles of 32 x 32 through shared memory) against the entry-by-entry
order of the named arrays, at the edges of the tiles.  The values are only moved: they are equal."""
import numpy as np
import pytest

from helpers import blocks, make_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["siam", "hubbard"])
@pytest.mark.parametrize("nK1,nK2,nK3", [(1, (1, 1), (1, 1)), (40, (16, 16), (16, 16)), (40, (17, 17), (17, 16)),
                                         (60, (33, 34), (3, 33)), (60, (34, 49), (33, 3))])
def test_round_trip(kind, nK1, nK2, nK3):
    cfg = dict(kind=kind, T=0.3, U=1.5, nG=nK1 + 4, nK1=nK1, nK2=nK2, nK3=nK3, mPi_factor=2)
    cfg.update(dict(e=0.2, Delta=0.5, D=10.0) if kind == "siam" else dict(mu=0.3, t1=1.0, t2=-0.2, L=3))
    rng = np.random.default_rng(nK1)
    gpu = make_gpu(cfg, False)
    n = gpu.flatten().size
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    gpu.unflatten(x)
    for name, s, e in blocks(cfg):
        got = gpu.get("Sigma" if name == "Sigma" else f"F.{name}")
        assert np.array_equal(np.ravel(got, order="F"), x[s:e])
    assert np.array_equal(gpu.flatten(), x)
    gpu.close()
