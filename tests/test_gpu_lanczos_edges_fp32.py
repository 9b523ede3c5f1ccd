"""The FP32 cluster Lanczos at the edges of its row splits: up to three rows per thread
(CTAs of 257, 512, 513, 768 and 769 rows, whose last rows' reads run past them), few rows,
and slices in global memory with short rows."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lanczos as olz
from oracle import maxcut as omaxcut
from oracle import rng as orng
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# n -> rows per CTA: 33 and 64 (one CTA), then 65, 128, 129, 256, 257, 512, 513, 768 and 769
# (sixteen); 438 rows of 80 entries and 312 of 120 do not fit beside the basis
@pytest.mark.parametrize("n,deg,inner", [(33, 4, 32), (64, 8, 20), (1040, 60, 32), (2048, 10, 32),
                                         (2064, 5, 24), (4096, 3, 32), (4112, 12, 32),
                                         (8192, 6, 32), (8208, 6, 32), (12_288, 4, 32),
                                         (12_304, 4, 31), (7000, 80, 32), (4990, 120, 32)])
def test_cluster_rows_fp32(cuda, n, deg, inner):
    from usbs_gb300 import _lib, api
    from usbs_gb300.problem import DeviceProblem, layout
    assert _lib.load().usbs_lanczos_kernel(n, inner, 32) == 1
    rng = np.random.default_rng(3)
    ne = max(1, int(round(deg * n / 2)))
    a = rng.integers(0, n, size=ne)
    b = (a + 1 + rng.integers(0, n - 1, size=ne)) % n
    W = wl.stream_adjacency(dict(n=n, i=np.minimum(a, b), j=np.maximum(a, b)))
    st, y, q0 = omaxcut.initialize_state(W, 4), rng.standard_normal(n), orng.default_q0(n)
    prob = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
    ov, _, ost = olz.eigsh_smallest(n, (-st.C).tocsr(), st.A_data, st.A_indices, y, q0, 3, inner,
                                    100, 1e-7)
    vals, vecs, info = api.eigsh_smallest(n, prob, None, None, y, q0, 3, inner, 100, 1e-5,
                                          c_scale=-1.0, precision=32, return_info=True)
    vals, vecs = vals.cpu().numpy(), vecs.double().cpu().numpy()
    assert info.status == 0 and ost["nconv"] >= 3
    scale = np.abs(ov).max()
    # the bounds of test_gpu_lanczos.py for FP32
    assert np.abs(vals - ov).max() < 1e-4 * scale
    Op = ((-st.C) + sp.diags(y)).tocsr()
    r = np.linalg.norm(Op @ vecs - vecs * vals[None, :], axis=0)
    assert r.max() < 1e-2 * scale
