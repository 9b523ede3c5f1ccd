"""The Lanczos paths at the edges of their rules: cluster slices in global memory
with short rows (four rows at a time, with a remainder), team-size problems one at a
time (full-GPU launches) against five at once (one shared launch), and the stream
path just above the shared-memory limit of x, whose first steps have fewer columns
than the dot kernel has column groups."""
import numpy as np
import pytest
import torch

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


# 313 and 312 rows a CTA whose entries (of 12 bytes) are beyond its shared memory; rows
# of 2 and 3 entries per lane; then x at and beyond the cluster's and the team's limits
# in FP64: 80 tiles of 256 rows, one row more (the stream path), 97 tiles
@pytest.mark.parametrize("n,deg,inner", [(5000, 60, 32), (4990, 90, 32), (12_100, 6, 32),
                                         (20_480, 4, 24), (20_481, 4, 32), (24_577, 6, 20)])
def test_paths_fp64(cuda, n, deg, inner):
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


# the two ways sum in the same order (the same teams), so the bits are the same
@pytest.mark.parametrize("n,deg,precision", [(12_033, 6, 64), (20_480, 4, 64), (17_000, 8, 32),
                                             (30_011, 12, 32)])
def test_team_size_alone_equals_shared(cuda, n, deg, precision):
    from usbs_gb300 import api
    from usbs_gb300.problem import DeviceProblem, layout
    st, y, q0 = _case(n, deg)
    prob = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
    alone = api.eigsh_smallest(n, prob, None, None, y, q0, 3, 32, 30, 1e-6, c_scale=-1.0,
                               precision=precision)
    shared = api.eigsh_smallest_batched([(prob, y, q0)] * 5, 3, 32, 30, 1e-6, c_scale=-1.0,
                                        precision=precision)
    for out in shared:
        assert torch.equal(alone[0], out[0]) and torch.equal(alone[1], out[1])
