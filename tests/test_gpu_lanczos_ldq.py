"""usbs_eigsh_smallest with leading dimensions of Q other than n rounded up to 32: odd
ones, and ones whose vectors would not fit the workspace if it followed them."""
import ctypes

import numpy as np
import pytest

from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _call(cuda, n, precision, ldq, guard=1 << 20):
    import torch
    from oracle import maxcut as omaxcut
    from usbs_gb300 import _lib
    from usbs_gb300.problem import DeviceProblem, layout
    lib = _lib.load()
    st = omaxcut.initialize_state(wl.er_graph(n, 3 * n, 5), 4)
    prob = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
    vt = torch.float64 if precision == 64 else torch.float32
    rs = np.random.default_rng(7)
    y = torch.tensor(rs.standard_normal(n), dtype=torch.float64, device=cuda)
    q = rs.standard_normal(n)
    q0 = torch.tensor(q / np.linalg.norm(q), dtype=vt, device=cuda)
    Q = torch.zeros((33, ldq), dtype=vt, device=cuda)
    evals = torch.zeros(3, dtype=torch.float64, device=cuda)
    info = torch.zeros(16, dtype=torch.int32, device=cuda)
    need = int(lib.usbs_eigsh_workspace_bytes(n, prob.nnz, 32, precision))
    ws = torch.full((need + guard,), 0xa5, dtype=torch.uint8, device=cuda)
    p = [ctypes.c_void_p(t.data_ptr()) for t in
         (prob.rowptr, prob.col, prob.c_val, prob.slot_ptr, prob.slot_tid, prob.t_con, prob.t_a0,
          y, q0, Q, evals, info, ws)]
    rc = lib.usbs_eigsh_smallest(n, prob.nnz, p[0], p[1], p[2], -1.0, *p[3:9], 3, 32, 6, 1e-6,
                                 precision, p[9], ldq, p[10], p[11], p[12], need,
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert bool((ws[need:] == 0xa5).all()), "written past the workspace"
    return rc, evals, Q[:3, :n].clone(), info[:6].clone()


# a cluster, a team's size in both precisions (odd n), and the stream path
@pytest.mark.parametrize("n,precision", [(1001, 64), (15_001, 64), (30_011, 32), (41_001, 32),
                                         (20_501, 64)])
def test_any_leading_dimension(cuda, n, precision):
    import torch
    stream = n > (40_960 if precision == 32 else 20_480)
    rc, vals, vecs, info = _call(cuda, n, precision, (n + 31) // 32 * 32)
    assert rc == 0 and int(info[5]) == 0
    step = 16 // (precision // 8)              # entries per 16 bytes
    for ldq in (n, n + 5000, (n // step + 1) * step, (n + 9000) // 32 * 32):
        r, v, V, i = _call(cuda, n, precision, ldq)
        if stream and ldq % step:
            assert r == -2
            continue
        assert r == 0
        assert torch.equal(v, vals) and torch.equal(V, vecs) and torch.equal(i, info)
