"""The cluster Lanczos at the edges of its row and column splits: CTAs of 1, 32,
33, 64, 65, 128, 129, 256 and 257 rows, short and long operator rows, an operator
slice that does not fit in shared memory, Krylov dimensions below 32."""
import numpy as np
import pytest

from oracle import lanczos as olz
from oracle import maxcut as omaxcut
from oracle import rng as orng
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _case(n, deg, seed=3):
    rng = np.random.default_rng(seed)
    ne = max(1, int(round(deg * n / 2)))
    a = rng.integers(0, n, size=ne)
    b = (a + 1 + rng.integers(0, n - 1, size=ne)) % n
    W = wl.stream_adjacency(dict(n=n, i=np.minimum(a, b), j=np.maximum(a, b)))
    return omaxcut.initialize_state(W, 4), rng.standard_normal(n), orng.default_q0(n)


# n -> rows per CTA with 64 wanted and at most 16 CTAs: 33, 64 (one CTA), 33
# (two), 64, 65, 128, 129, 256, 257 (sixteen); the last has 120-entry rows whose slices
# (two thirds of a megabyte a CTA) are read from global memory
@pytest.mark.parametrize("n,deg,inner", [(33, 4, 32), (64, 8, 32), (66, 40, 20), (1024, 3, 32),
                                         (1040, 60, 32), (2048, 10, 32), (2064, 5, 24),
                                         (4096, 3, 32), (4112, 12, 32), (4500, 120, 32)])
def test_cluster_rows_fp64(cuda, n, deg, inner):
    from usbs_gb300 import api
    from usbs_gb300.problem import DeviceProblem, layout
    st, y, q0 = _case(n, deg)
    prob = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
    args = (q0, 3, inner, 100, 1e-9)
    ov, oV, ost = olz.eigsh_smallest(n, (-st.C).tocsr(), st.A_data, st.A_indices, y, *args)
    gv, gV, info = api.eigsh_smallest(n, prob, None, None, y, *args, c_scale=-1.0, precision=64,
                                      return_info=True)
    assert info.status == 0 and info.num_converged >= 3 and ost["nconv"] >= 3
    gv, gV = gv.cpu().numpy(), gV.cpu().numpy()
    np.testing.assert_allclose(gv, ov, rtol=1e-9, atol=1e-9 * np.abs(ov).max())
    for j in range(3):
        assert abs(gV[:, j] @ oV[:, j]) > 1 - 1e-10, j

