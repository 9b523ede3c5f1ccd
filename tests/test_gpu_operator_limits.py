"""The operator callbacks at the largest sizes that the entry points take: 2^31 - 1
pattern entries, rows, constraints or triples, where a position plus a grid's stride no
longer fits 32 signed bits.  About 45 GB on the device."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

LIM = 2 ** 31 - 1


def _lib(cuda):
    import torch
    from usbs_gb300 import _lib as L
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("less than 60 GB of device memory free")
    return torch, L, L.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def test_assemble_and_apply(cuda):
    torch, L, lib, st = _lib(cuda)
    c_val = torch.ones(LIM, dtype=torch.float64, device=cuda)
    c_val[-3:] = torch.tensor([2.0, 5.0, -7.0], dtype=torch.float64, device=cuda)
    out = torch.empty(LIM, dtype=torch.float32, device=cuda)
    none = _p(None)
    L.check(lib.usbs_assemble_operator(LIM, _p(c_val), -1.0, none, none, none, none, none,
                                       _p(out), 32, st), "usbs_assemble_operator")
    assert out[-3:].tolist() == [-2.0, -5.0, 7.0]
    assert bool((out[:-3] == -1.0).all())
    # rows of 2048 entries, the last one short of that by one: sums of ones are exact
    n = 2 ** 20
    rowptr = (torch.arange(n + 1, dtype=torch.int64, device=cuda) * 2048).clamp_(max=LIM).int()
    col = torch.zeros(LIM, dtype=torch.int32, device=cuda)
    x = torch.ones(n, dtype=torch.float32, device=cuda)
    want = torch.full((n,), -2048.0, device=cuda)
    want[-1] = -(2047.0 - 3.0)                       # 2047 entries, of which 2 + 5 - 7 = 0
    y = torch.zeros(n, dtype=torch.float32, device=cuda)
    L.check(lib.usbs_operator_apply(n, LIM, _p(rowptr), _p(col), _p(out), _p(x), _p(y), 32, st),
            "usbs_operator_apply")
    assert torch.equal(y, want)
    y.zero_()
    L.check(lib.usbs_operator_apply_direct(n, LIM, _p(rowptr), _p(col), _p(c_val), -1.0, none,
                                           none, none, none, none, _p(x), _p(y), 32, st),
            "usbs_operator_apply_direct")
    assert torch.equal(y, want)


# one constraint of two triples at each end, the others empty
def test_constraints(cuda):
    torch, L, lib, st = _lib(cuda)
    con_ptr = torch.full((LIM + 1,), 2, dtype=torch.int32, device=cuda)
    con_ptr[0] = 0
    con_ptr[-1] = 4
    i32 = dict(dtype=torch.int32, device=cuda)
    f64 = dict(dtype=torch.float64, device=cuda)
    t_row, t_col = torch.tensor([0, 1, 0, 1], **i32), torch.tensor([0, 1, 1, 0], **i32)
    t_a, U = torch.tensor([1.0, 2.0, 3.0, 4.0], **f64), torch.tensor([3.0, 5.0], **f64)
    out = torch.full((LIM,), -1.0, **f64)
    L.check(lib.usbs_apply_A_operator(LIM, 1, _p(con_ptr), _p(t_row), _p(t_col), _p(t_a), _p(U), 2,
                                      _p(out), st), "usbs_apply_A_operator")
    assert out[0].item() == 59.0 and out[-1].item() == 105.0
    assert not bool(out[1:-1].any())


# the same by rows: n = 2^31 - 1 rows, of which the first and the last have triples
def test_adjoint(cuda):
    torch, L, lib, st = _lib(cuda)
    row_ptr = torch.full((LIM + 1,), 2, dtype=torch.int32, device=cuda)
    row_ptr[0] = 0
    row_ptr[-1] = 4
    i32 = dict(dtype=torch.int32, device=cuda)
    f64 = dict(dtype=torch.float64, device=cuda)
    r_con, r_col = torch.tensor([0, 1, 0, 1], **i32), torch.tensor([0, LIM - 1, LIM - 1, 0], **i32)
    r_a, z = torch.tensor([1.0, 2.0, 3.0, 4.0], **f64), torch.tensor([0.5, 0.25], **f64)
    U = torch.zeros(LIM, **f64)
    U[0], U[-1] = 3.0, 5.0
    out = torch.full((LIM,), -1.0, **f64)
    L.check(lib.usbs_apply_A_adjoint(LIM, 1, _p(row_ptr), _p(r_con), _p(r_col), _p(r_a), _p(z),
                                     _p(U), LIM, _p(out), LIM, st), "usbs_apply_A_adjoint")
    assert out[0].item() == 4.0 and out[-1].item() == 10.5
    assert not bool(out[1:-1].any())


# one long constraint and row: the last thousand of 2^31 - 1 triples
def test_last_triples(cuda):
    torch, L, lib, st = _lib(cuda)
    ptr = torch.tensor([LIM - 1000, LIM], dtype=torch.int32, device=cuda)
    idx = torch.zeros(LIM, dtype=torch.int32, device=cuda)
    a = torch.ones(LIM, dtype=torch.float64, device=cuda)
    two = torch.full((1,), 2.0, dtype=torch.float64, device=cuda)
    out = torch.zeros(1, dtype=torch.float64, device=cuda)
    L.check(lib.usbs_apply_A_adjoint(1, 1, _p(ptr), _p(idx), _p(idx), _p(a), _p(two), _p(two), 1,
                                     _p(out), 1, st), "usbs_apply_A_adjoint")
    assert out.item() == 4000.0
    out.zero_()
    L.check(lib.usbs_apply_A_operator(1, 1, _p(ptr), _p(idx), _p(idx), _p(a), _p(two), 1, _p(out),
                                      st), "usbs_apply_A_operator")
    assert out.item() == 4000.0
