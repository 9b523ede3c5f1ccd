"""The constraint callbacks at the line between the thread and the warp path, and
the assembled operator's values, bit for bit."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import operators as oops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 5, 11])
def test_constraint_lengths(cuda, k):
    """Constraints and rows of 0, 1, 2, 7, 8, 9, 31, 32, 33, 64, 127, 129 and 1000 triples."""
    from usbs_gb300 import api
    from usbs_gb300.problem import DeviceProblem, layout
    rng = np.random.default_rng(5)
    sizes = [0, 1, 2, 7, 8, 9, 31, 32, 33, 64, 127, 129, 1000, 8, 0, 1]
    m, n = len(sizes), 40
    con = np.repeat(np.arange(m), sizes)
    # rows of the same lengths: row i holds sizes[i] triples (rows 16.. none)
    row = rng.permutation(np.repeat(np.arange(m), sizes))
    idx = np.stack([con, row, rng.integers(0, n, con.size)], 1)
    a = rng.standard_normal(con.size)
    prob = DeviceProblem(layout(sp.csr_matrix((n, n)), a, idx, m=m), cuda)
    U, z = rng.standard_normal((n, k)), rng.standard_normal(m)
    got = api.apply_A_operator_batched(m, None, None, U, problem=prob).cpu().numpy()
    np.testing.assert_allclose(got, oops.apply_A_operator_batched(m, a, idx, U), rtol=1e-12,
                               atol=1e-12)
    got = api.apply_A_adjoint_batched(n, None, None, z, U, problem=prob).cpu().numpy()
    np.testing.assert_allclose(got, oops.apply_A_adjoint_batched(n, a, idx, z, U), rtol=1e-12,
                               atol=1e-12)


# entries: below and above the four-per-thread line (311,296)
@pytest.mark.parametrize("n,per_row", [(300, 7), (50_000, 8)])
@pytest.mark.parametrize("scale", [1.0, -1.0, 0.37, 0.0])
def test_assembled_values(cuda, n, per_row, scale):
    """out = scale C + A*(w) on the pattern: FP64, and its rounding to FP32 (subnormal,
    overflowing, infinite and tied values among C's)."""
    import torch
    from usbs_gb300 import _lib
    from usbs_gb300.problem import DeviceProblem, layout
    rng = np.random.default_rng(n)
    i = np.repeat(np.arange(n), per_row)
    j = rng.integers(0, n, i.size)
    C = sp.csr_matrix((np.ones(i.size), (i, j)), shape=(n, n))
    C.sum_duplicates()
    v = rng.standard_normal(C.nnz) * 10.0 ** rng.integers(-50, 42, C.nnz)
    ties = rng.random(C.nnz) < 0.2           # halfway between two floats
    v[ties] = np.float64(np.float32(rng.standard_normal(ties.sum()))) * (1 + 2.0 ** -24)
    v[:6] = [0.0, -0.0, np.inf, -np.inf, 3.4028235677973366e38, 1e-46]
    C.data[:] = v
    d = rng.permutation(n)[: n // 2]          # diagonal triples on half of the rows, two on some
    d = np.concatenate([d, d[: n // 8]])
    idx = np.stack([np.arange(d.size), d, d], 1)
    a, w = rng.standard_normal(d.size), rng.standard_normal(d.size)
    h = layout(C, a, idx, m=d.size)
    p = DeviceProblem(h, cuda)
    ref = scale * h.c_val if scale else np.zeros(h.nnz)
    for q in np.nonzero(np.diff(h.slot_ptr))[0]:
        for t in h.slot_tid[h.slot_ptr[q]:h.slot_ptr[q + 1]]:
            ref[q] += h.t_a0[t] * w[h.t_con[t]]       # (the device uses one FMA)
    plain = np.diff(h.slot_ptr) == 0
    lib, wt = _lib.load(), torch.as_tensor(w, device=cuda)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())     # noqa: E731
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for prec, dt in ((64, torch.float64), (32, torch.float32)):
        out = torch.empty(h.nnz, dtype=dt, device=cuda)
        _lib.check(lib.usbs_assemble_operator(h.nnz, ptr(p.c_val), scale, ptr(p.slot_ptr),
                                              ptr(p.slot_tid), ptr(p.t_con), ptr(p.t_a0), ptr(wt),
                                              ptr(out), prec, st), "usbs_assemble_operator")
        got = out.cpu().numpy()
        with np.errstate(all="ignore"):
            want = ref if prec == 64 else ref.astype(np.float32)
        assert np.array_equal(got[plain], want[plain])
        fin = ~plain & np.isfinite(want) & (np.abs(ref) < 1e30)
        np.testing.assert_allclose(got[fin], want[fin], rtol=1e-14 if prec == 64 else 1e-6,
                                   atol=1e-14 if prec == 64 else 1e-6)
