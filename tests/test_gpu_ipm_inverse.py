"""The interior-point kernel's Gauss-Jordan inverse: against 64-bit inverses, and its
report of pivots that are zero or infinite (the solve's status bit 8)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inverse(cuda, A):
    import torch
    from usbs_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    a = torch.tensor(A, dtype=torch.float64, device=cuda)
    inv = torch.zeros_like(a)
    ok = torch.full((1,), -1, dtype=torch.int32, device=cuda)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (a, inv, ok)]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.usbs_selftest_inverse(n, *p, st), "usbs_selftest_inverse")
    return inv.cpu().numpy(), int(ok.item())


@pytest.mark.parametrize("n", [1, 2, 5, 11, 12])
def test_inverse(cuda, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 3.0 * np.eye(n)[rng.permutation(n)]   # rows exchanged
    inv, ok = _inverse(cuda, A)
    assert ok == 1
    # Gauss-Jordan with partial pivoting: n eps cond^2 with room
    c = np.linalg.cond(A)
    assert np.abs(inv @ A - np.eye(n)).max() <= 10 * n * c * c * 2.0 ** -53


@pytest.mark.parametrize("value,flagged", [(np.inf, True), (-np.inf, True), (0.0, True),
                                           (1.7e308, False), (5e-324, False)])
@pytest.mark.parametrize("n", [1, 3, 11])
def test_unusable_pivots_are_reported(cuda, n, value, flagged):
    A = np.diag(np.linspace(1.0, 2.0, n))
    A[n // 2, n // 2] = value
    _, ok = _inverse(cuda, A)
    assert ok == (0 if flagged else 1)
