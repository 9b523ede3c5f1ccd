"""The interior-point kernel's reciprocal against the IEEE division, and outer
iterations at bundle sizes whose Newton systems cross its register blocks."""
import numpy as np
import pytest

from oracle import maxcut as omaxcut
from oracle import rng as orng
from oracle import usbs as ousbs
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def test_reciprocal_bits(cuda):
    """Bit for bit 1/x: random bit patterns (every exponent, both signs), mantissas next
    to powers of two, zeros, infinities, NaN and subnormals."""
    import ctypes

    import torch
    from usbs_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(11)
    bits = rng.integers(0, 2 ** 64, size=4_000_000, dtype=np.uint64)
    near = rng.integers(0, 64, size=1_000_000, dtype=np.uint64)
    top = np.uint64(2 ** 52 - 1)
    near = np.where(rng.random(near.size) < 0.5, near, top - near)
    expo = rng.integers(0, 4096, size=near.size, dtype=np.uint64) << np.uint64(52)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.3e-308, 1.8e308, 1.0, -2.0,
                        2.0 ** -1022, 2.0 ** 1023, 1.5 * 2.0 ** 1022, 1.5 * 2.0 ** 1021])
    x = np.concatenate([bits.view(np.float64), (expo | near).view(np.float64), special])
    xt = torch.as_tensor(x, device=cuda)
    y = torch.empty_like(xt)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (xt, y)]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.usbs_selftest_recip(x.size, p[0], p[1], st), "usbs_selftest_recip")
    got = y.cpu().numpy()
    with np.errstate(all="ignore"):
        ref = 1.0 / x
    fin = ~np.isnan(ref)
    assert np.array_equal(np.isnan(got), ~fin)
    assert np.array_equal(got[fin].view(np.uint64), ref[fin].view(np.uint64))


# svec orders 3, 10 and 36: one, one and two blocks of 32 (three: the largest bundle of
# test_gpu_usbs.py)
@pytest.mark.parametrize("k_curr,k_past", [(2, 0), (4, 0), (4, 4)])
def test_first_iteration_1e9(cuda, k_curr, k_past):
    from usbs_gb300 import solver
    S = wl.MAXCUT_SETTINGS
    st = omaxcut.initialize_state(wl.er_graph(300, 4000, 7), 10)
    n = st.C.shape[0]
    q0 = orng.default_q0(n)
    otr = []
    a = (st, n, n, 2.0 * n, 2.0, S["rho"], S["beta"], k_curr, k_past, 1, np.inf, -1.0, -1.0, -1.0,
         32, 200, 1e-9, S["subprob_max_iters"])
    ousbs.usbs(*a, q0=q0, trace=otr)
    gtr = solver.usbs(*a, 1.0, None, None, None, q0=q0, precision=64, return_trace=True)[1]
    for key in ("primal_obj", "obj_ub", "lb_spec_est", "pen_dual_obj", "cand_pen_dual_obj",
                "tr_X"):
        x, y = otr[0][key], gtr[0][key]
        assert abs(x - y) <= 1e-9 * max(1.0, abs(x), abs(y)), (key, x, y)
