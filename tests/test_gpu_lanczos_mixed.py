"""Lanczos batches that mix problems of one cluster's size with larger ones, and small
problems without the cluster path: every problem keeps its loop state and partial sums
apart, whatever its size, so its results are those of the oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import lanczos as olz
from oracle import maxcut as omaxcut
from oracle import rng as orng
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

# the bounds of test_gpu_lanczos.py: eigenvalues, then residuals, of the operator's scale
EIG = {64: 1e-9, 32: 1e-4}
RES = {64: 1e-6, 32: 1e-2}
TOL = {64: 1e-9, 32: 1e-5}


def _case(n, deg=6.0, seed=3):
    rng = np.random.default_rng(seed + n)
    ne = max(1, int(round(deg * n / 2)))
    a = rng.integers(0, n, size=ne)
    b = (a + 1 + rng.integers(0, n - 1, size=ne)) % n
    W = wl.stream_adjacency(dict(n=n, i=np.minimum(a, b), j=np.maximum(a, b)))
    return omaxcut.initialize_state(W, 4), rng.standard_normal(n), orng.default_q0(n)


def _check(case, out, precision, pairs, inner, restarts):
    st, y, q0 = case
    n = st.C.shape[0]
    ov, _, ost = olz.eigsh_smallest(n, (-st.C).tocsr(), st.A_data, st.A_indices, y, q0, pairs,
                                    inner, restarts, TOL[precision])
    vals, vecs, info = out
    vals, vecs = vals.cpu().numpy(), vecs.double().cpu().numpy()
    assert info.status == 0 and info.num_converged >= pairs and ost["nconv"] >= pairs
    scale = np.abs(ov).max()
    assert np.abs(vals - ov).max() < EIG[precision] * scale, n
    Op = ((-st.C) + sp.diags(y)).tocsr()
    r = np.linalg.norm(Op @ vecs - vecs * vals[None, :], axis=0)
    assert r.max() < RES[precision] * scale, n


# beside the last problem of each batch, which does not, the others would fit a
# cluster; 41,000 (FP32) and 20,481 (FP64) rows take the stream path
@pytest.mark.parametrize("precision,sizes", [
    (32, (100, 30_011)), (32, (200, 41_000)), (32, (100, 200, 41_000)), (32, (33, 256)),
    (32, (257, 30_011)), (64, (60, 15_000)), (64, (128, 20_480)), (64, (129, 12_100)),
    (64, (100, 20_481)), (64, (300, 15_000, 20_481))])
def test_mixed_batch(cuda, precision, sizes):
    from usbs_gb300 import api
    from usbs_gb300.problem import DeviceProblem, layout
    cases = [_case(n) for n in sizes]
    probs = [(DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=st.C.shape[0]), cuda), y, q0)
             for st, y, q0 in cases]
    out = api.eigsh_smallest_batched(probs, 3, 32, 60, TOL[precision], c_scale=-1.0,
                                     precision=precision, return_info=True)
    for case, o in zip(cases, out):
        _check(case, o, precision, 3, 32, 60)


# run by the test below in a process of its own: the switch is read once per process
def _without_clusters():
    import torch
    from oracle import usbs as ousbs
    from usbs_gb300 import _lib, api, solver
    from usbs_gb300.problem import DeviceProblem, layout
    cuda = torch.device("cuda:0")
    for precision in (64, 32):
        for n in (33, 100, 200, 300, 5200):
            assert _lib.load().usbs_lanczos_kernel(n, 32, precision) == 0
            case = _case(n)
            st, y, q0 = case
            prob = DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda)
            out = api.eigsh_smallest(n, prob, None, None, y, q0, 3, 32, 60, TOL[precision],
                                     c_scale=-1.0, precision=precision, return_info=True)
            _check(case, out, precision, 3, 32, 60)
    # one outer iteration, the cooperative path and the one without cooperative launches
    S = wl.MAXCUT_SETTINGS
    st = omaxcut.initialize_state(wl.er_graph(120, 900, 7), 10)
    n = st.C.shape[0]
    a = (st, n, n, 2.0 * n, 2.0, S["rho"], S["beta"], 4, 1, 1, np.inf, -1.0, -1.0, -1.0, 32, 200,
         1e-9, S["subprob_max_iters"])
    otr = []
    ousbs.usbs(*a, q0=orng.default_q0(n), trace=otr)
    for path in (0, 2):
        gtr = solver.usbs(*a, 1.0, None, None, None, q0=orng.default_q0(n), precision=64,
                          return_trace=True, lanczos_path=path)[1]
        for key in ("primal_obj", "obj_ub", "pen_dual_obj", "tr_X"):
            x, y = otr[0][key], gtr[0][key]
            assert abs(x - y) <= 1e-9 * max(1.0, abs(x), abs(y)), (path, key, x, y)


def test_small_problems_without_clusters(cuda):
    env = dict(os.environ, USBS_LANCZOS_CLUSTER="0")
    r = subprocess.run([sys.executable, "-c", "from tests.test_gpu_lanczos_mixed import "
                        "_without_clusters as f; f()"], env=env, timeout=300,
                       capture_output=True, text=True,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-3000:]
