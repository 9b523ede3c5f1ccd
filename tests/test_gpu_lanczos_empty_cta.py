"""Cluster batches whose smallest problem has fewer rows than its clusters' CTAs times
their rows: CTAs past its last row own none and start past the end of its arrays.  The
arrays end where their memory does not (rowptr is the head of a longer tensor whose rest
would be far out of range as an offset)."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lanczos as olz
from oracle import maxcut as omaxcut
from oracle import rng as orng
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("sizes", [(5000, 20), (5000, 33, 9), (700, 17)])
def test_ctas_without_rows(cuda, sizes, precision):
    import torch
    from usbs_gb300 import api
    from usbs_gb300.problem import DeviceProblem, layout
    probs, refs = [], []
    for n in sizes:
        inner = min(min(sizes), 32)
        st = omaxcut.initialize_state(wl.er_graph(n, min(3 * n, n * (n - 1) // 2), 5), 4)
        p = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
        tail = torch.full((4096,), 0x7fffff00, dtype=torch.int32, device=cuda)
        p.rowptr = torch.cat([p.rowptr, tail])[:n + 1]
        y, q0 = np.random.default_rng(n).standard_normal(n), orng.default_q0(n)
        probs.append((p, y, q0))
        refs.append((st, y, q0))
    tol = 1e-9 if precision == 64 else 1e-5
    out = api.eigsh_smallest_batched(probs, 2, inner, 200, tol, c_scale=-1.0, precision=precision,
                                     return_info=True)
    for (st, y, q0), (vals, vecs, info) in zip(refs, out):
        n = st.C.shape[0]
        ov, _, ost = olz.eigsh_smallest(n, (-st.C).tocsr(), st.A_data, st.A_indices, y, q0, 2,
                                        inner, 200, tol)
        vals, vecs = vals.cpu().numpy(), vecs.double().cpu().numpy()
        scale = np.abs(ov).max()
        assert info.status == 0 and ost["nconv"] >= 2
        assert np.abs(vals - ov).max() < (1e-9 if precision == 64 else 1e-4) * scale
        Op = ((-st.C) + sp.diags(y)).tocsr()
        r = np.linalg.norm(Op @ vecs - vecs * vals[None, :], axis=0)
        assert r.max() < (1e-6 if precision == 64 else 1e-2) * scale
