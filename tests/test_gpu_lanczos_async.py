"""Team-size Lanczos calls (one launch, or the launches of a bounded number of cycles
followed by it): they return before a busy stream gets to them, fill the info words, and
give the shared launch's bits also where that launch takes over in mid-solve."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from oracle import maxcut as omaxcut
from oracle import rng as orng
from usbs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _problem(cuda, n, zero=False):
    from usbs_gb300.problem import DeviceProblem, layout
    if zero:
        C, A, I = sp.csr_matrix((n, n)), np.ones(n), np.stack([np.arange(n)] * 3, 1)
        return (DeviceProblem(layout(C, A, I, m=n), cuda), torch.zeros(n, dtype=torch.float64,
                                                                       device=cuda),
                orng.default_q0(n))
    st = omaxcut.initialize_state(wl.er_graph(n, 3 * n, 5), 4)
    y = np.random.default_rng(n).standard_normal(n)
    return (DeviceProblem(layout(st.C, st.A_data, st.A_indices, m=n), cuda),
            torch.as_tensor(y, device=cuda), orng.default_q0(n))


def _dev(problem, precision):
    p, y, q0 = problem
    vt = torch.float64 if precision == 64 else torch.float32
    return p, y, torch.as_tensor(np.asarray(q0), dtype=vt, device=y.device)


@pytest.mark.parametrize("n,precision", [(15_000, 64), (30_011, 32)])
def test_returns_while_the_stream_is_busy(cuda, n, precision):
    from usbs_gb300 import _lib, api
    assert _lib.load().usbs_lanczos_kernel(n, 32, precision) == 0
    prob = _dev(_problem(cuda, n), precision)

    def one():
        return api.eigsh_smallest(n, prob[0], None, None, prob[1], prob[2], 10, 32, 10, 1e-7,
                                  c_scale=-1.0, precision=precision)

    def two():
        return api.eigsh_smallest_batched([prob, prob], 10, 32, 10, 1e-7, c_scale=-1.0,
                                          precision=precision)

    for call in (one, two):
        call()                                       # (kernels loaded)
        torch.cuda.synchronize()
        torch.cuda._sleep(2_000_000_000)             # about a second of a waiting stream
        busy = torch.cuda.Event()
        busy.record()
        out = call()
        assert not busy.query()
        torch.cuda.synchronize()
        del out


@pytest.mark.parametrize("n,precision", [(15_000, 64), (30_011, 32)])
def test_info_words(cuda, n, precision):
    from usbs_gb300 import api
    p, y, q0 = _dev(_problem(cuda, n), precision)
    _, _, i = api.eigsh_smallest(n, p, None, None, y, q0, 10, 32, 10, 1e-7, c_scale=-1.0,
                                 precision=precision, return_info=True)
    red, a, b, c = i.phase_kcycles[1:]
    assert min(red, a, b, c, i.restart_kcycles, i.eig_kcycles) > 0
    assert i.total_kcycles >= red + a + b + c + i.restart_kcycles - 6     # (each rounded down)


# 40 restarts are more than are planned ahead; on the zero operator every step breaks
# down, and from two restarts on the cycles no longer have the planned number of steps;
# with all vectors wanted a restart drops none, so the later cycles have no steps
@pytest.mark.parametrize("n,precision,zero,pairs,inner,restarts", [
    (15_000, 64, False, 10, 32, 40), (30_011, 32, False, 10, 32, 40), (12_100, 64, False, 3, 24, 2),
    (15_000, 64, True, 4, 32, 3), (30_011, 32, True, 4, 32, 3), (30_011, 32, False, 8, 8, 4),
    (12_100, 64, False, 2, 5, 60), (12_100, 64, False, 1, 32, 1), (12_100, 64, False, 1, 32, 0)])
def test_equals_the_shared_launch(cuda, n, precision, zero, pairs, inner, restarts):
    from usbs_gb300 import api
    prob = _dev(_problem(cuda, n, zero), precision)
    kw = dict(c_scale=-1.0, precision=precision, return_info=True)
    tol = 1e-12
    alone = api.eigsh_smallest(n, prob[0], None, None, prob[1], prob[2], pairs, inner, restarts,
                               tol, **kw)
    pair = api.eigsh_smallest_batched([prob] * 2, pairs, inner, restarts, tol, **kw)
    shared = api.eigsh_smallest_batched([prob] * 4, pairs, inner, restarts, tol, **kw)
    for out in pair + [alone]:
        ref = shared[0]
        if restarts:
            assert torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])
        for w in ("k_saved", "num_converged", "restarts", "breakdowns", "matvecs", "status",
                  "sum_active_columns", "sum_saved"):
            assert getattr(out[2], w) == getattr(ref[2], w), w
    assert not zero or alone[2].breakdowns > 0
