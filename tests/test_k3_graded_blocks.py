"""The K3 contractions of blocks below Nν3 = 32 and the adjoint's up to it (fdga_k3_mma.cu, the default there) on
operands graded against each other: A falls along ω by 2^39 as M rises, so that every term of an output counts alike although A's row and
M's column hold entries 2^39 apart.  The FP64 CUDA-core GEMMs (option k3_fp64_tensor_cores = 0) do not see the
grading; the digit products hold an entry relative to the largest of its row or column.

F0's p-channel corrections are r(ν) c(ω) times phases with r rising, c = 1/r: C(ν, ν') = r(ν) c(ν') O(1), and the
outputs are compared divided by their grading.  frule: dA graded like A.  rrule: ȳ(ν, ν') = c(ν) r(ν') times
phases, Ā(ν, ω) = c(ν) r(ω) O(1).
Tolerance: two FP64 sums of at most 32 complex products, 2 · 72 · 2^-53 of the sum of their magnitudes, that sum
at most 32 times the largest output: 5e-13.  At Nν3 = 32 the map's digits are relative to row and column bounds (they
were relative to a block's before they had rows and columns), and only the adjoint is compared."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _phases(rng, *shape):
    return np.exp(2j * np.pi * rng.random(shape))


@pytest.mark.parametrize("n", [4, 7, 12, 16])
def test_graded_operands(n):
    import fdgasolver as F
    rng = np.random.default_rng(n)
    N, nO, T = 2 * n, 2, 0.3
    NO = 2 * nO - 1
    r = 2.0 ** (39 * np.arange(N) / (N - 1))
    c = 1 / r
    graded = lambda: r[None, :, None] * c[None, None, :] * _phases(rng, NO, N, N)  # noqa: E731  [Ω, ν, ν']
    nG = n + 6
    Gb = F.siam_bare_Green(T, nG, Delta=0.5, e=0.2, D=10.0)
    S = F.ParquetSolver(n + 4, (nO, n + 1), (nO, n), Gb, 0 * Gb, 0 * Gb, F.RefVertex(T, 1.5, graded(), graded()),
                        mPi_factor=4)
    n1, n2, n3 = 2 * (n + 4) - 1, NO * 2 * (n + 1), NO * N * N
    k3 = slice(n1 + n2, n1 + n2 + n3)  # γp's K3, flattened [Ω, ν, ν'] (Ω fastest)
    part = lambda x: x[k3].reshape(N, N, NO).transpose(2, 1, 0)  # noqa: E731

    def full(a):
        x = np.zeros(S.state_len, dtype=complex)
        x[k3] = a.transpose(2, 1, 0).reshape(-1)
        return x

    v = full(graded())
    yb = full(c[None, :, None] * r[None, None, :] * _phases(rng, NO, N, N))
    out = []
    for opt in (0, 2):
        S.set_option("k3_fp64_tensor_cores", opt)
        f = part(S.fixed_point(full(np.zeros((NO, N, N)))))
        S.unflatten(full(np.zeros((NO, N, N))))
        jv = part(S.frule(v)[1])
        S.unflatten(full(np.zeros((NO, N, N))))
        xb = part(S.rrule(yb)[1])
        out.append((f / r[None, :, None] / c[None, None, :], jv / r[None, :, None] / c[None, None, :],
                    xb / c[None, :, None] / r[None, None, :]))
    for a, b in list(zip(*out))[2 if N == 32 else 0:]:
        assert np.abs(a).max() > 0
        assert np.abs(b - a).max() < 5e-13 * np.abs(a).max()
    S.close()
