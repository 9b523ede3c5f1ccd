"""reconstruct_from_sketch where the two largest singular values of P agree to a few
digits, or all: rho = sqrt(n) eps ||P||_2 is formed in FP64, so Lambda is that of a
64-bit evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sketch(n, s, gap, seed):
    """Omega and P whose Omega^T P is symmetric positive definite; the squares of P's
    singular values are 1, 1 / (1 + gap), then 0.64 and less."""
    rng = np.random.default_rng(seed)
    Q, _ = np.linalg.qr(rng.standard_normal((n, 2 * s)))
    W, _ = np.linalg.qr(rng.standard_normal((s, s)))
    sv = np.concatenate([[1.0, 1.0 / np.sqrt(1.0 + gap)], np.linspace(0.8, 0.3, s)[:s - 2]])[:s]
    B = rng.standard_normal((s, s)) / np.sqrt(s)
    return (Q[:, :s] + Q[:, s:] @ B) @ W.T, (Q[:, :s] * sv) @ W.T


def _lambda(Om, P, eps):
    """utils/common.py:99-116 in 64 bits."""
    rho = np.sqrt(P.shape[0]) * eps * np.linalg.svd(P, compute_uv=False)[0]
    Pr = P + rho * Om
    B = Om.T @ Pr
    M = np.linalg.solve(np.linalg.cholesky(0.5 * (B + B.T)), Pr.T)
    return np.maximum(np.linalg.svd(M, compute_uv=False) ** 2 - rho, 0.0)


# eps = 0.01 makes Lambda feel rho: a relative error of 1e-9 in lambda_max is one of 3e-11
# there.  The systems have condition below 100 and order at most 32: round-off of at most
# 32 * 100 * 2^-53 = 4e-13
@pytest.mark.parametrize("gap", [0.0, 1e-10, 1e-8, 3e-8, 1e-7, 3e-7, 1e-3])
@pytest.mark.parametrize("s", [2, 10, 17, 32])
def test_lambda_of_nearly_equal_singular_values(cuda, gap, s):
    from usbs_gb300 import rounding
    for seed in range(4):
        Om, P = _sketch(400, s, gap, seed)
        ref = _lambda(Om, P, 1e-2)
        _, lam = rounding.reconstruct_from_sketch(Om, P, approx_eps=1e-2, device=cuda)
        assert np.abs(lam.cpu().numpy() - ref).max() <= 1e-12 * ref.max(), seed
