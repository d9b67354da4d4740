"""The sums of the Krylov iteration (fixed grid of 608 x 256 threads, one finishing warp a sum) at the edges of
that grid: the residual norm that the device reports against the one of the returned x."""
import numpy as np
import pytest

from fhhos4_gb300 import hho


# unknowns: 130 (one CTA, a part of it), 816 (four CTAs), 37,184 (146), 305,920 (two rounds of the grid),
# 993,024 (a second group of four rounds)
SIZES = [(5, 1), (12, 1), (56, 3), (160, 3), (288, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32", "df"])
@pytest.mark.parametrize("n,k", SIZES)
def test_gpu_reported_residual_is_the_residual_of_x(n, k, precision):
    """Three FCG iterations. Tolerance: the reported norm is that of the recursive residual, which leaves
    b - A x by the rounding of x and of three updates (2^-47 in pairs) times |A| |x| / |b|."""
    pytest.importorskip("torch")
    from fhhos4_gb300 import solver as S
    As, Ps, b, bs = hho.generate(2, n, k)
    s = S.fcg_mg(As, Ps, bs, precision=precision, maxit=3, tol=1e-30)
    x = s.Solve(b)
    true = np.linalg.norm(b - As[0] @ x) / np.linalg.norm(b)
    scale = np.linalg.norm(abs(As[0]) @ np.abs(x)) / np.linalg.norm(b)
    assert abs(s.History[-1] - true) <= 64 * 2.0 ** -47 * scale
    s.Context().close()
