"""The one-pass operator product is the assembled operator's, bit for bit: lane counts 1
to 32, rows of every length (none at all included), with and without dual weights, scales
that are and are not signs."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("avg", [1.0, 4.0, 9.0, 20.0, 42.0, 90.0])      # 1, 2, 4, 8, 16, 32 lanes
def test_same_bits(cuda, avg, precision):
    import torch
    from usbs_gb300 import _lib
    from usbs_gb300.problem import DeviceProblem, layout
    rng = np.random.default_rng(int(avg))
    n = 523                                    # no multiple of any lane group or block
    lens = np.minimum(rng.integers(0, int(2 * avg) + 1, n), n)
    lens[:3] = [0, 1, min(int(4 * avg), n)]
    lens[-1] = 0
    i = np.repeat(np.arange(n), lens)
    j = np.concatenate([rng.choice(n, k, replace=False) for k in lens] + [np.zeros(0, int)])
    C = sp.csr_matrix((rng.standard_normal(i.size), (i, j.astype(int))), shape=(n, n))
    # triples on a third of the pattern, several on some entries
    pick = rng.integers(0, i.size, i.size // 3)
    idx = np.stack([rng.integers(0, 50, pick.size), i[pick], j.astype(int)[pick]], 1)
    p = DeviceProblem(layout(C, rng.standard_normal(pick.size), idx, m=50), cuda)
    vt = torch.float64 if precision == 64 else torch.float32
    it = torch.int64 if precision == 64 else torch.int32
    x = torch.as_tensor(rng.standard_normal(n), dtype=vt, device=cuda)
    lib, st = _lib.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)     # noqa: E731
    for w in (None, torch.as_tensor(rng.standard_normal(50), device=cuda)):
        for scale in (0.0, 1.0, -1.0, 0.37):
            op = torch.empty(p.nnz, dtype=vt, device=cuda)
            two, one = torch.empty(n, dtype=vt, device=cuda), torch.empty(n, dtype=vt, device=cuda)
            _lib.check(lib.usbs_assemble_operator(
                p.nnz, ptr(p.c_val), scale, ptr(p.slot_ptr), ptr(p.slot_tid), ptr(p.t_con),
                ptr(p.t_a0), ptr(w), ptr(op), precision, st), "usbs_assemble_operator")
            _lib.check(lib.usbs_operator_apply(n, p.nnz, ptr(p.rowptr), ptr(p.col), ptr(op), ptr(x),
                                               ptr(two), precision, st), "usbs_operator_apply")
            _lib.check(lib.usbs_operator_apply_direct(
                n, p.nnz, ptr(p.rowptr), ptr(p.col), ptr(p.c_val), scale, ptr(p.slot_ptr),
                ptr(p.slot_tid), ptr(p.t_con), ptr(p.t_a0), ptr(w), ptr(x), ptr(one), precision,
                st), "usbs_operator_apply_direct")
            assert torch.equal(one.view(it), two.view(it)), (scale, w is None)
