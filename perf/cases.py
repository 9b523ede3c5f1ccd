"""What a user of this package has it do, as measurable cases.

Each case is a plain dict: ``kind`` names the public entry point, the rest its
sizes, precision and options.  ``prepare`` makes what a program holds before the
call (problem data and handles resident on the device), ``run`` is the call.

Inputs: MaxCut operators C = L/4 of Erdos-Renyi graphs (the serving stream's
generator), +-1 toruses and 6-nearest-neighbour geometric graphs, QAP
relaxations on a 10 x 10 grid; dual vectors and start vectors are drawn from the
seed.  Graphs of up to 50,000 nodes are drawn from the seed too; larger graphs
and the QAP instances are one fixed instance per size (as benchmark instances
are), kept on the host between preparations because laying them out takes
seconds.
"""
import functools

import numpy as np
import scipy.sparse as sp
import torch

from usbs_gb300 import api, rounding, solver
from usbs_gb300 import workloads as wl
from usbs_gb300.problem import DeviceProblem, layout
from usbs_gb300.problems import maxcut, qap

SEEDED_NODES = 50_000      # larger graphs are one fixed instance per size
INNER, RESTARTS, TOL = 32, 10, 1e-7   # the Lanczos budget of the reference's settings
EXACT_NODES = 3000         # dense eigenvalues up to here


def listed():
    """The listed cases."""
    return [
        # the operator callback on a Gset-scale graph: one small launch chain
        dict(name="apply_er800_fp64", kind="apply", graph="er", n=800, deg=48.0, precision=64),
        # the same callback on the large sparse instance
        dict(name="apply_rgg1m_fp32", kind="apply", graph="rgg", n=1_000_000, deg=6.0,
             precision=32),
        # A(V V^T) and A*(z) V of the QAP relaxation (3.4e5 constraints) at its bundle size
        dict(name="constraints_qap30", kind="constraints", problem="qap", l=30, k=2),
        # the plain FP64 eigensolve at Gset scale
        dict(name="eigsh_er800_fp64", kind="eigsh", graph="er", n=800, deg=48.0, precision=64,
             pairs=10),
        # the mixed-precision eigensolve of the 100 x 100 spin-glass torus
        dict(name="eigsh_torus10k_fp32", kind="eigsh", graph="torus", n=10_000, deg=4.0,
             precision=32, pairs=10),
        # a mid-size request of the serving stream
        dict(name="eigsh_er30k_fp32", kind="eigsh", graph="er", n=30_011, deg=12.0, precision=32,
             pairs=10),
        # the large sparse instance
        dict(name="eigsh_rgg1m_fp32", kind="eigsh", graph="rgg", n=1_000_000, deg=6.0,
             precision=32, pairs=10),
        # many small requests at once
        dict(name="eigsh_batch48_fp32", kind="eigsh_batch", count=48, n_lo=500, n_hi=5000,
             precision=32, pairs=10),
        # outer iterations from a cold start: spin glass, mixed precision
        dict(name="usbs_torus10k_mixed", kind="usbs", graph="torus", n=10_000, deg=4.0,
             precision=32, iters=5),
        # outer iterations from a cold start: Gset scale, plain FP64
        dict(name="usbs_er800_fp64", kind="usbs", graph="er", n=800, deg=48.0, precision=64,
             iters=5),
        # outer iterations of the QAP relaxation, mixed precision
        dict(name="usbs_qap30_mixed", kind="usbs_qap", l=30, precision=32, iters=4),
        # the rounding callback at a condition check
        dict(name="round_torus10k", kind="round", graph="torus", n=10_000, deg=4.0, s=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def _graph_of(rng, lo, hi):
    """A graph family and an odd or even size of it in [lo, hi]."""
    n = _log_int(rng, lo, hi)
    g = rng.choice(["er", "er", "torus", "rgg"]) if n <= SEEDED_NODES else "rgg"
    if g == "torus":
        side = max(3, int(np.sqrt(n)))
        return dict(graph=g, n=side * side, deg=4.0)
    return dict(graph=g, n=n, deg=round(rng.uniform(4.0, 40.0), 1) if g == "er" else 6.0)


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["apply", "constraints", "eigsh", "eigsh", "eigsh", "eigsh_batch", "usbs",
                       "usbs", "usbs_qap", "round"])
    prec = rng.choice([32, 64])
    if kind == "apply":
        return dict(kind=kind, precision=prec, **_graph_of(rng, 200, 1_000_000))
    if kind == "constraints":
        if rng.random() < 0.5:
            return dict(kind=kind, problem="qap", l=rng.randint(6, 30), k=rng.randint(1, 3))
        return dict(kind=kind, problem="maxcut", n=_log_int(rng, 200, 300_000),
                    k=rng.randint(1, 11))
    if kind == "eigsh":
        hi = 1_000_000 if prec == 32 else 300_000
        return dict(kind=kind, precision=prec, pairs=rng.choice([1, 5, 10]),
                    **_graph_of(rng, 200, hi))
    if kind == "eigsh_batch":
        lo = rng.choice([200, 500])
        return dict(kind=kind, count=rng.randint(2, 48), n_lo=lo, n_hi=_log_int(rng, 1000, 5000),
                    precision=prec, pairs=rng.choice([5, 10]))
    if kind == "usbs":
        return dict(kind=kind, precision=prec, iters=rng.randint(1, 4),
                    **_graph_of(rng, 200, 8_000))
    if kind == "usbs_qap":
        return dict(kind=kind, l=rng.randint(6, 30), precision=prec, iters=rng.randint(1, 3))
    return dict(kind=kind, s=rng.choice([4, 8, 10]), **_graph_of(rng, 200, 200_000))


# ---------------------------------------------------------------- inputs

def _adjacency(graph, n, deg, seed):
    if graph == "torus":
        return wl.torus_graph(int(round(np.sqrt(n))), seed)
    if graph == "rgg":
        return wl.rgg_knn_graph(n, int(deg), seed)
    rng = np.random.default_rng(seed)
    ne = int(round(deg * n / 2))
    a = rng.integers(0, n, size=ne)
    b = (a + 1 + rng.integers(0, n - 1, size=ne)) % n
    return wl.stream_adjacency(dict(n=n, i=np.minimum(a, b), j=np.maximum(a, b)))


def _layout_of(graph, n, deg, seed):
    C = maxcut.objective(_adjacency(graph, n, deg, seed))
    A_data, A_idx, _, _ = maxcut.problem_data(C.shape[0])
    return layout(C, A_data, A_idx, m=C.shape[0])


@functools.lru_cache(maxsize=3)
def _fixed_layout(graph, n, deg):
    return _layout_of(graph, n, deg, 0)


@functools.lru_cache(maxsize=2)
def _qap_state(l):
    D, W = wl.qap_instance(l, 0)
    st = qap.initialize_state(D, W, l)
    return st, solver.host_problem_layout(st)


def _host_layout(case, seed):
    if case["n"] > SEEDED_NODES:
        return _fixed_layout(case["graph"], case["n"], case["deg"])
    return _layout_of(case["graph"], case["n"], case["deg"], seed)


def _normal(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _dual(n, seed):
    """A dual vector as the outer iteration has one: entries of order 0.5."""
    return 0.5 * _normal(seed, n)


def _unit(n, seed):
    q = _normal(seed + 1_000_003, n)
    return q / q.norm()


def _dtype(precision):
    return torch.float64 if precision == 64 else torch.float32


def _batch_sizes(case, seed):
    """Sizes of a batch's problems: the same for every seed, so that a pass costs the same."""
    rng = np.random.default_rng(case["count"])
    n = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), case["count"]))
    return [int(v) for v in n], [float(d) for d in rng.uniform(4.0, 40.0, case["count"])]


def _eigsh_inputs(case, seed):
    """(host layout, dual vector, start vector) of a single eigsh case."""
    h = _host_layout(case, seed)
    return h, _dual(h.n, seed), _unit(h.n, seed)


def _sketch(n, s, seed):
    """Omega and P = X Omega of a near-optimal X = F F^T with unit diagonal and rank 11."""
    F = _normal(seed + 1, n, 11) * (0.7 ** torch.arange(11, device="cuda", dtype=torch.float64))
    F /= F.norm(dim=1, keepdim=True)
    Om = _normal(seed + 2, s, n).t()          # columns contiguous, as the solver keeps them
    return Om, (F @ (F.t() @ Om)).t().contiguous().t()


def prepare(case, seed):
    """Problem data, handles and vectors, resident on the device."""
    kind = case["kind"]
    if kind == "apply":
        h, w, x = _eigsh_inputs(case, seed)
        return dict(case=case, prob=DeviceProblem(h, "cuda"), w=w,
                    x=x.to(_dtype(case["precision"])))
    if kind == "eigsh":
        h, w, q0 = _eigsh_inputs(case, seed)
        return dict(case=case, prob=DeviceProblem(h, "cuda"), w=w,
                    q0=q0.to(_dtype(case["precision"])))
    if kind == "eigsh_batch":
        ns, degs = _batch_sizes(case, seed)
        probs = []
        for i, (n, deg) in enumerate(zip(ns, degs)):
            p = DeviceProblem(_layout_of("er", n, deg, seed + i), "cuda")
            probs.append((p, _dual(n, seed + i), _unit(n, seed + i).to(_dtype(case["precision"]))))
        return dict(case=case, probs=probs)
    if kind == "constraints":
        if case["problem"] == "qap":
            st, h = _qap_state(case["l"])
        else:
            A_data, A_idx, _, _ = maxcut.problem_data(case["n"])
            h = layout(sp.csr_matrix((case["n"], case["n"])), A_data, A_idx, m=case["n"])
        k = case["k"]
        V = _normal(seed, k, h.n).t() / np.sqrt(h.n)
        return dict(case=case, prob=DeviceProblem(h, "cuda"), V=V, z=_dual(h.m, seed))
    if kind == "usbs":
        W = _adjacency(case["graph"], case["n"], case["deg"], seed)
        st = maxcut.initialize_state(W, wl.MAXCUT_SETTINGS["sketch_dim"])
        return dict(case=case, st=st, inst=solver.DeviceInstance(st, "cuda"),
                    q0=_unit(st.C.shape[0], seed))
    if kind == "usbs_qap":
        st, h = _qap_state(case["l"])
        return dict(case=case, st=st, inst=solver.DeviceInstance(st, "cuda", h),
                    q0=_unit(st.C.shape[0], seed))
    C = maxcut.objective(_adjacency(case["graph"], case["n"], case["deg"],
                                    seed if case["n"] <= SEEDED_NODES else 0))
    Om, P = _sketch(C.shape[0], case["s"], seed)
    return dict(case=case, C=rounding.DeviceCSR(C), Om=Om, P=P)


# ---------------------------------------------------------------- calls

def _usbs(state, n, m, trace_ub, rho, k_curr, k_past):
    c, S = state["case"], wl.MAXCUT_SETTINGS
    out, info = solver.usbs(state["st"], n, m, trace_ub, S["trace_factor"], rho, S["beta"],
                            k_curr, k_past, c["iters"], np.inf, 1e-7, 1e-7, 1e-7, INNER, RESTARTS,
                            S["subprob_eps"], S["subprob_max_iters"], q0=state["q0"],
                            precision=c["precision"], instance=state["inst"], return_info=True)
    return dict(y=out.y, z=out.z, P=out.P, V=info["V"], tr_X=out.tr_X,
                primal_obj=out.primal_obj, obj_gap=info["obj_gap"],
                infeas_gap=info["infeas_gap"])


def run(state):
    """One call of the case's entry point."""
    c = state["case"]
    kind = c["kind"]
    if kind == "apply":
        return api.operator_apply(state["prob"], -1.0, state["w"], state["x"], c["precision"])
    if kind == "eigsh":
        p = state["prob"]
        return api.eigsh_smallest(p.n, p, None, None, state["w"], state["q0"], c["pairs"], INNER,
                                  RESTARTS, TOL, c_scale=-1.0, precision=c["precision"])
    if kind == "eigsh_batch":
        got = api.eigsh_smallest_batched(state["probs"], c["pairs"], INNER, RESTARTS, TOL,
                                         c_scale=-1.0, precision=c["precision"])
        return dict(values=torch.stack([e for e, _ in got]),
                    vectors=torch.cat([v for _, v in got]))
    if kind == "constraints":
        p = state["prob"]
        return (api.apply_A_operator_batched(p.m, None, None, state["V"], problem=p),
                api.apply_A_adjoint_batched(p.n, None, None, state["z"], state["V"], problem=p))
    if kind == "usbs":
        n, S = state["st"].C.shape[0], wl.MAXCUT_SETTINGS
        return _usbs(state, n, n, 2.0 * n, S["rho"], S["k_curr"], S["k_past"])
    if kind == "usbs_qap":
        st, S = state["st"], wl.QAP_SETTINGS
        return _usbs(state, st.C.shape[0], st.b.shape[0], 2.0 * (c["l"] + 1) * st.SCALE_X,
                     S["rho"], S["k_curr"], S["k_past"])
    E, lam = rounding.reconstruct_from_sketch(state["Om"], state["P"])
    value, columns, signs = rounding.max_cut_values(state["P"], state["Om"], state["C"])
    return dict(E=E, lam=lam, value=value, columns=columns, signs=signs)


# ---------------------------------------------------------------- work and exact values

def _nnz(n, deg):
    return n * (deg + 1)


def _qap_counts(l):
    """(lifted order, pattern entries, constraints, triples), nearly."""
    off = l * l * (l - 1) ** 2
    return l * l + 1, off + 3 * l * l + 2 * l ** 3, off / 2 + 3 * l * l, off + 9 * l * l + 4 * l ** 3


def _eigsh_work(n, nnz, vt, pairs, steps=None):
    """Operator, dual and start vector in, pairs out; a thick-restart cycle keeps
    about two thirds of the basis, so a later cycle has about a third of the steps."""
    steps = INNER + (RESTARTS - 1) * INNER // 3 if steps is None else steps
    return dict(bytes=nnz * 12 + n * (4 + 8 + vt) + pairs * n * vt,
                flops=steps * (2 * nnz + 8 * n * 24) + RESTARTS * 2 * n * INNER * 21)


def _iteration_work(n, nnz, vt, k, s, m):
    """One outer iteration: one eigensolve, the projections and Grams over V, the
    interior-point systems (about 50 Newton steps of order k (k + 1) / 2)."""
    e = _eigsh_work(n, nnz, vt, k)
    sv = k * (k + 1) // 2
    return dict(bytes=e["bytes"] + 8 * (n * (2 * k + 3 * s) + 6 * m),
                flops=e["flops"] + 2 * nnz * k + m * sv * sv + 6 * n * k * k +
                50 * (2 * sv ** 3 / 3 + 20 * sv ** 2))


def work(case):
    """Bytes each read or written once, and operations, of one pass."""
    kind = case["kind"]
    vt = 8 if case.get("precision", 64) == 64 else 4
    if kind in ("apply", "eigsh"):
        n, nnz = case["n"], _nnz(case["n"], case["deg"])
        if kind == "eigsh":
            return _eigsh_work(n, nnz, vt, case["pairs"])
        return dict(bytes=nnz * 12 + n * (4 + 8 + 2 * vt), flops=2 * nnz + 2 * n)
    if kind == "eigsh_batch":
        w = [_eigsh_work(n, _nnz(n, d), vt, case["pairs"]) for n, d in zip(*_batch_sizes(case, 0))]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    if kind == "constraints":
        if case["problem"] == "qap":
            n, _, m, t = _qap_counts(case["l"])
        else:
            n = m = t = case["n"]
        k = case["k"]
        return dict(bytes=2 * t * 16 + m * (4 + 8 + 8) + n * (4 + 16 * k), flops=6 * t * k)
    if kind == "usbs":
        w = _iteration_work(case["n"], _nnz(case["n"], case["deg"]), vt, 11, 10, case["n"])
    elif kind == "usbs_qap":
        n, nnz, m, _ = _qap_counts(case["l"])
        w = _iteration_work(n, nnz, vt, 2, case["l"], m)
    else:
        n, s = case["n"], case["s"]
        return dict(bytes=2 * 16 * n * s + 8 * n * s + 16 * n * (case["deg"] + 1),
                    flops=2 * (3 * 2 * n * s * s + 2 * n * s * s) + 2 * s * n * case["deg"])
    return dict(bytes=w["bytes"] * case["iters"], flops=w["flops"] * case["iters"])


def _csr(h, w):
    """-C + A*(w) of a diagonal-constraint layout, in 64 bits on the host."""
    C = sp.csr_matrix((h.c_val, h.col, h.rowptr), shape=(h.n, h.n))
    return (sp.diags(w) - C).tocsr()


def _rounding_exact(Om, P, C, eps=1e-6):
    """Sketch reconstruction and cut values (Tropp et al. 2017, Algorithm 3)."""
    n, s = P.shape
    rho = np.sqrt(n) * eps * np.linalg.norm(P, 2)
    P = P + rho * Om
    B = Om.T @ P
    L = np.linalg.cholesky(0.5 * (B + B.T))
    E, sv, _ = np.linalg.svd(np.linalg.solve(L, P.T).T, full_matrices=False)
    Wm = np.where(E > 0, 1.0, -1.0)
    cuts = np.einsum("ij,ij->j", Wm, C @ Wm)
    return np.clip(sv ** 2 - rho, 0.0, None), cuts


def exact(case, seed):
    """What run() computes, in 64 bits by numpy, scipy or torch; None where there is no
    value that does not depend on the start (eigenvectors, whole solves)."""
    kind = case["kind"]
    if kind == "apply":
        h, w, x = _eigsh_inputs(case, seed)
        x = x.to(_dtype(case["precision"])).double().cpu().numpy()
        return _csr(h, w.cpu().numpy()) @ x
    if kind in ("eigsh", "eigsh_batch"):
        if kind == "eigsh":
            if case["n"] > EXACT_NODES:
                return None
            hs = [_eigsh_inputs(case, seed)]
        else:
            ns, degs = _batch_sizes(case, seed)
            if sum(n ** 3 for n in ns) > 8 * EXACT_NODES ** 3:
                return None
            hs = [(_layout_of("er", n, d, seed + i), _dual(n, seed + i), None)
                  for i, (n, d) in enumerate(zip(ns, degs))]
        vals = []
        for h, w, _ in hs:
            A = torch.as_tensor(_csr(h, w.cpu().numpy()).toarray(), device="cuda")
            vals.append(torch.linalg.eigvalsh(A)[:case["pairs"]].cpu().numpy())
        return (vals[0], None) if kind == "eigsh" else dict(values=np.stack(vals), vectors=None)
    if kind == "constraints":
        s = prepare(case, seed)
        h, V, z = s["prob"].host, s["V"].cpu().numpy(), s["z"].cpu().numpy()
        con = np.repeat(np.arange(h.m), np.diff(h.con_ptr))
        a = h.t_a * np.einsum("tk,tk->t", V[h.t_row], V[h.t_col])
        A = sp.csr_matrix((h.r_a * z[h.r_con], h.r_col, h.row_ptr), shape=(h.n, h.n))
        return np.bincount(con, weights=a, minlength=h.m), A @ V
    if kind == "round":
        s = prepare(case, seed)
        C = sp.csr_matrix((s["C"].val.cpu().numpy(), s["C"].col.cpu().numpy(),
                           s["C"].rowptr.cpu().numpy()))
        lam, cuts = _rounding_exact(s["Om"].cpu().numpy(), s["P"].cpu().numpy(), C)
        return dict(E=None, lam=lam, value=cuts.max(), columns=cuts, signs=None)
    return None
