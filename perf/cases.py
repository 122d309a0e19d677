"""Performance cases of the solve engine: the calls its users make, over the
range of sizes they make them at.

Every case is one call (or one forward + backward) of a public entry point:
``linear_solve`` with the LU, Cholesky, QR and GMRES solvers, the batched and
ragged solves, GMRES-IR, batched CG on the Poisson stencil and the solve
server.  Matrices have the distributions of the benchmark configurations:
G/sqrt(n) + I for LU, G Gᵀ/n + 1e-2 I for Cholesky, i.i.d. N(0, 1) for least
squares, U diag(sigma) Vᵀ with log-spaced sigma for GMRES-IR.
"""

import math

import torch

import lineax_gb300 as lx
from lineax_gb300 import _krylov, batched, mixed, serve

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # one small dense system: what a Newton step or a filter update in a
        # host program calls, bound by launches and host latency
        {"name": "lu_solve_48", "kind": "lu_solve", "n": 48},
        # the ordinary dense solve of a simulation or a fit
        {"name": "lu_solve_1000", "kind": "lu_solve", "n": 1000},
        # the vmapped solve of the plain-LU benchmark configuration
        {"name": "lu_batch_64x128", "kind": "lu_batch", "batch": 64, "n": 128, "k": 1},
        # a solve inside a differentiated program: value, then the gradients
        # of the matrix and the right-hand side (odd order)
        {"name": "lu_grad_2003", "kind": "lu_grad", "n": 2003},
        # a covariance or kernel matrix (tagged positive definite, odd order)
        {"name": "chol_solve_1531", "kind": "chol_solve", "n": 1531},
        # a regression with a few hundred coefficients, in FP64
        {"name": "qr_lstsq_3001x401", "kind": "qr_lstsq", "m": 3001, "n": 401},
        # the ragged SPD batch of the headline benchmark, data resident
        {"name": "spd_ragged_4096", "kind": "spd_ragged", "count": 4096, "nmin": 16,
         "nmax": 512, "kmax": 8},
        # the large dense system of the mixed-precision LU configuration
        {"name": "gmres_ir_8192", "kind": "gmres_ir", "n": 8192, "k": 16, "cond": 100.0},
        # the least-squares configuration (mixed-precision QR)
        {"name": "qr_mixed_16384x2048", "kind": "qr_mixed", "m": 16384, "n": 2048},
        # the batched matrix-free CG configuration, a block of its iterations
        {"name": "cg_poisson_2048_64rhs", "kind": "cg_poisson", "nx": 2048, "ny": 2048, "k": 64,
         "steps": 32},
        # a restarted Krylov solve of a dense nonsymmetric operator
        {"name": "gmres_dense_2000", "kind": "gmres_dense", "n": 2000},
        # the served stream: mixed kinds and orders, 30 % on a known operator
        {"name": "serve_96", "kind": "serve", "count": 96, "nmax": 4096, "mix": 7},
    ]


def _log(rng, lo, hi):
    return int(min(hi, max(lo, math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["lu_solve", "lu_batch", "lu_grad", "chol_solve", "qr_lstsq", "spd_ragged",
                       "gmres_ir", "qr_mixed", "cg_poisson", "gmres_dense", "serve"])
    if kind == "lu_solve":
        return {"kind": kind, "n": _log(rng, 24, 2500)}
    if kind == "lu_batch":
        return {"kind": kind, "batch": _log(rng, 8, 512), "n": rng.randint(16, 168),
                "k": rng.randint(1, 4)}
    if kind == "lu_grad":
        return {"kind": kind, "n": _log(rng, 64, 2500)}
    if kind == "chol_solve":
        return {"kind": kind, "n": _log(rng, 64, 2500)}
    if kind == "qr_lstsq":
        n = _log(rng, 24, 512)
        return {"kind": kind, "m": min(8192, int(n * math.exp(rng.uniform(0.0, math.log(16.0))))),
                "n": n}
    if kind == "spd_ragged":
        nmax = _log(rng, 64, 512)
        return {"kind": kind, "count": _log(rng, 128, 4096), "nmin": rng.randint(8, 32),
                "nmax": nmax, "kmax": rng.randint(1, 8)}
    if kind == "gmres_ir":
        return {"kind": kind, "n": 4 * _log(rng, 200, 1800), "k": rng.randint(1, 16),
                "cond": float(10 ** rng.uniform(1.0, 2.0))}
    if kind == "qr_mixed":
        n = _log(rng, 128, 2048)
        return {"kind": kind, "m": 4 * (_log(rng, 2 * n, min(8 * n, 16384)) // 4), "n": n}
    if kind == "cg_poisson":
        nx, ny = _log(rng, 200, 2048), _log(rng, 200, 2048)
        kmax = max(1, min(64, (1 << 27) // (nx * ny)))
        return {"kind": kind, "nx": nx, "ny": ny, "k": _log(rng, 1, kmax), "steps": 32}
    if kind == "gmres_dense":
        return {"kind": kind, "n": _log(rng, 200, 3000)}
    return {"kind": "serve", "count": rng.randint(24, 80), "nmax": _log(rng, 512, 2500),
            "mix": rng.randint(0, 10 ** 6)}


# -- inputs -------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _randn(g, *shape, dtype=F64):
    return torch.randn(*shape, dtype=dtype, device=DEV, generator=g)


def _lu_matrix(g, n, *batch, scale=1.0):
    a = _randn(g, *batch, n, n) * (scale / math.sqrt(n))
    a.diagonal(dim1=-2, dim2=-1).add_(1.0)
    return a


def _spd_matrix(g, n):
    x = _randn(g, n, n)
    a = x @ x.T / n
    a.diagonal().add_(1e-2)
    return a


def _conditioned(g, n, cond):
    """U diag(sigma) Vᵀ with orthogonal U, V and sigma log-spaced in
    [1/cond, 1] (FP32 factors: their rounding does not move the condition
    number)."""
    def orthogonal():
        return torch.linalg.qr(_randn(g, n, n, dtype=torch.float32))[0]

    u, v = orthogonal(), orthogonal()
    sig = torch.logspace(0, -math.log10(cond), n, dtype=torch.float32, device=DEV)
    return ((u * sig) @ v.T).to(F64).contiguous()


def _ragged_sizes(case):
    """Orders and right-hand-side counts of a ragged batch: part of the case,
    not of the seed (log-uniform orders, uniform counts)."""
    g = torch.Generator().manual_seed(case["count"] * 1009 + case["nmax"])
    u = torch.rand(case["count"], generator=g, dtype=F64)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"] + 1)
    n = torch.exp(lo + (hi - lo) * u).floor().clamp(case["nmin"], case["nmax"]).long()
    k = torch.randint(1, case["kmax"] + 1, (case["count"],), generator=g)
    n, order = torch.sort(n, descending=True)
    return n.tolist(), k[order].tolist()


def _serve_plan(case):
    """(kind, operator id, order, right-hand sides, fresh) of every request."""
    g = torch.Generator().manual_seed(case["mix"])
    u = torch.rand(case["count"], 5, generator=g, dtype=F64).tolist()
    plan, ops = [], []
    for reuse, which, size, pick, rhs in u:
        k = 1 + int(16 * rhs)
        if ops and reuse < 0.3:
            op = int(pick * len(ops))
            plan.append((ops[op][0], op, ops[op][1], k, False))
            continue
        kind = "lu" if which < 0.5 else ("cholesky" if which < 0.8 else "qr")
        n = int(min(case["nmax"], math.exp(math.log(32) + size * math.log((case["nmax"] + 1) / 32))))
        plan.append((kind, len(ops), n, k, True))
        ops.append((kind, n))
    return plan


def _serve_data(case, seed):
    g = _gen(seed)
    plan, mats, rhs = _serve_plan(case), {}, []
    for kind, op, n, k, fresh in plan:
        if fresh:
            # 0.8 G: condition numbers of tens, so that the tolerance of the
            # server and not the matrices' conditioning sets the error
            mats[op] = _spd_matrix(g, n) if kind == "cholesky" else _lu_matrix(g, n, scale=0.8)
        rhs.append(_randn(g, k, n))
    return plan, mats, rhs


def _ragged_data(case, seed):
    g = _gen(seed)
    n_list, k_list = _ragged_sizes(case)
    a = torch.empty(sum(n * n for n in n_list), dtype=F64, device=DEV)
    b = _randn(g, sum(n * k for n, k in zip(n_list, k_list)))
    x = _randn(g, a.numel())
    o = 0
    for n in n_list:
        m = x[o: o + n * n].view(n, n)
        d = a[o: o + n * n].view(n, n)
        torch.mm(m, m.T, out=d)
        d.div_(n).diagonal().add_(1e-2)
        o += n * n
    return a, b, n_list, k_list


def _data(case, seed):
    """The tensors a case's call takes."""
    g, kind = _gen(seed), case["kind"]
    if kind in ("lu_solve", "lu_grad"):
        a = _lu_matrix(g, case["n"])
        return a, _randn(g, case["n"]), _randn(g, case["n"])
    if kind == "lu_batch":
        return (_lu_matrix(g, case["n"], case["batch"]),
                _randn(g, case["batch"], case["k"], case["n"]))
    if kind == "chol_solve":
        return _spd_matrix(g, case["n"]), _randn(g, case["n"])
    if kind == "gmres_dense":
        n = case["n"]
        a = _randn(g, n, n) * (0.5 / math.sqrt(n))
        a.diagonal().add_(1.0)
        return a, _randn(g, n)
    if kind == "gmres_ir":
        return _conditioned(g, case["n"], case["cond"]), _randn(g, case["k"], case["n"])
    if kind in ("qr_lstsq", "qr_mixed"):
        m, n = case["m"], case["n"]
        a = _randn(g, m, n, dtype=torch.float32).to(F64)
        return a, a @ _randn(g, n) + 1e-3 * _randn(g, m)
    if kind == "cg_poisson":
        return (_randn(g, case["k"], case["nx"] * case["ny"]),)
    raise ValueError(kind)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        plan, mats, rhs = _serve_data(case, seed)
        host = {op: a.cpu().pin_memory() for op, a in mats.items()}
        reqs = [serve.Request(rid, knd, rhs[rid].cpu().pin_memory(), op, host[op] if fresh else None)
                for rid, (knd, op, n, k, fresh) in enumerate(plan)]
        return {"kind": kind, "requests": reqs}
    if kind == "spd_ragged":
        a, b, n_list, k_list = _ragged_data(case, seed)
        rb = batched.RaggedBatch.from_packed(a, b, n_list, k_list, DEV)
        ws = batched.MixedWorkspace(rb.batch, rb.max_n, rb.max_nrhs, DEV)
        return {"kind": kind, "batch": rb, "workspace": ws}
    data = _data(case, seed)
    state = {"kind": kind, "data": data}
    if kind == "lu_grad":
        a, b, ct = data
        a.requires_grad_(True)
        b.requires_grad_(True)
        state.update(op=lx.MatrixLinearOperator(a), solver=lx.LU())
    elif kind == "lu_solve":
        state.update(op=lx.MatrixLinearOperator(data[0]), solver=lx.LU())
    elif kind == "chol_solve":
        state.update(op=lx.MatrixLinearOperator(data[0], lx.positive_semidefinite_tag),
                     solver=lx.Cholesky())
    elif kind == "qr_lstsq":
        state.update(op=lx.MatrixLinearOperator(data[0]), solver=lx.QR())
    elif kind == "qr_mixed":
        state.update(op=lx.MatrixLinearOperator(data[0]), solver=lx.QR(precision="mixed"))
    elif kind == "gmres_dense":
        state.update(op=lx.MatrixLinearOperator(data[0]), solver=lx.GMRES(rtol=1e-10, atol=1e-10))
    elif kind == "cg_poisson":
        state.update(op=lx.Poisson2DOperator(case["nx"], case["ny"]), steps=case["steps"])
    return state


def run(state):
    kind = state["kind"]
    if kind in ("lu_solve", "chol_solve", "qr_lstsq", "qr_mixed", "gmres_dense"):
        return lx.linear_solve(state["op"], state["data"][1], state["solver"]).value
    if kind == "lu_grad":
        a, b, ct = state["data"]
        x = lx.linear_solve(state["op"], b, state["solver"]).value
        ga, gb = torch.autograd.grad(x, (a, b), ct)
        return [x.detach(), ga, gb]
    if kind == "lu_batch":
        x, info = batched.lu_solve_batched(*state["data"])
        return [x, info]
    if kind == "spd_ragged":
        res = batched.spd_solve_ragged_mixed(state["batch"], workspace=state["workspace"])
        return [res.x, res.info]
    if kind == "gmres_ir":
        return mixed.gmres_ir(*state["data"], restart=8).x
    if kind == "cg_poisson":
        return _krylov.cg_poisson_mixed(state["op"], state["data"][0], rtol=1e-10, atol=1e-10,
                                        max_steps=state["steps"]).y
    out = serve.SolveServer(DEV).run(state["requests"], realtime=False)
    return torch.cat([c.x.reshape(-1) for c in out])


# -- what a pass cannot do without --------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("lu_solve", "lu_grad"):
        n = case["n"]
        if kind == "lu_solve":
            return {"bytes": 8 * (n * n + 2 * n), "flops": 2 * n ** 3 / 3 + 2 * n * n}
        # the matrix in, its gradient out; two solves and an outer product
        return {"bytes": 8 * (2 * n * n + 5 * n), "flops": 2 * n ** 3 / 3 + 5 * n * n}
    if kind == "lu_batch":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * case["batch"] * (n * n + 2 * n * k),
                "flops": case["batch"] * (2 * n ** 3 / 3 + 2 * n * n * k)}
    if kind == "chol_solve":
        n = case["n"]
        return {"bytes": 8 * (n * n + 2 * n), "flops": n ** 3 / 3 + 2 * n * n}
    if kind in ("qr_lstsq", "qr_mixed"):
        m, n = case["m"], case["n"]
        return {"bytes": 8 * (m * n + m + n), "flops": 2 * m * n * n - 2 * n ** 3 / 3 + 4 * m * n}
    if kind == "spd_ragged":
        n_list, k_list = _ragged_sizes(case)
        return {"bytes": sum(8 * n * n + 16 * n * k for n, k in zip(n_list, k_list)),
                "flops": sum(n ** 3 / 3 + 4 * n * n * k for n, k in zip(n_list, k_list))}
    if kind == "gmres_ir":
        n, k = case["n"], case["k"]
        return {"bytes": 8 * (n * n + 2 * n * k), "flops": 2 * n ** 3 / 3 + 4 * n * n * k}
    if kind == "cg_poisson":
        # b in, x out, and per iteration the direction, the residual and the
        # iterate of FP32 iterations read and written once
        pts = case["nx"] * case["ny"] * case["k"]
        return {"bytes": pts * (16 + 24 * case["steps"]), "flops": pts * 19 * case["steps"]}
    if kind == "gmres_dense":
        # the Gram-Schmidt cycles' products with the operator (about 40)
        n = case["n"]
        return {"bytes": 8 * (n * n + 2 * n), "flops": 40 * 2 * n * n}
    flops = nbytes = 0
    for knd, op, n, k, fresh in _serve_plan(case):
        nbytes += 16 * n * k + (8 * n * n if fresh else 0)
        flops += 2 * n * n * k
        if fresh:
            flops += n ** 3 * {"lu": 2 / 3, "cholesky": 1 / 3, "qr": 4 / 3}[knd]
    return {"bytes": nbytes, "flops": flops}


# -- the same results in 64 bits, without the engine ---------------------------


def _poisson(x, nx, ny):
    """The 5-point negative Laplacian of flattened nx × ny grids (ny fastest)
    with zero boundaries."""
    g = x.view(-1, nx, ny)
    y = 4.0 * g
    y[:, 1:, :] -= g[:, :-1, :]
    y[:, :-1, :] -= g[:, 1:, :]
    y[:, :, 1:] -= g[:, :, :-1]
    y[:, :, :-1] -= g[:, :, 1:]
    return y.view_as(x)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        plan, mats, rhs = _serve_data(case, seed)
        return torch.cat([torch.linalg.solve(mats[op], rhs[i].T).T.reshape(-1)
                          for i, (knd, op, n, k, fresh) in enumerate(plan)])
    if kind == "spd_ragged":
        a, b, n_list, k_list = _ragged_data(case, seed)
        out, oa, ob = torch.empty_like(b), 0, 0
        for n, k in zip(n_list, k_list):
            s = a[oa: oa + n * n].view(n, n)
            out[ob: ob + n * k].view(k, n).copy_(
                torch.linalg.solve(s, b[ob: ob + n * k].view(k, n).T).T)
            oa, ob = oa + n * n, ob + n * k
        return [out, None]
    data = _data(case, seed)
    if kind == "lu_grad":
        a, b, ct = data
        lu, piv = torch.linalg.lu_factor(a)
        x = torch.linalg.lu_solve(lu, piv, b[:, None])[:, 0]
        z = torch.linalg.lu_solve(lu, piv, ct[:, None], adjoint=True)[:, 0]
        return [x, -torch.outer(z, x), z]
    if kind in ("lu_solve", "chol_solve", "gmres_dense"):
        return torch.linalg.solve(data[0], data[1])
    if kind == "lu_batch":
        return [torch.linalg.solve(data[0], data[1].mT).mT.contiguous(), None]
    if kind == "gmres_ir":
        return torch.linalg.solve(data[0], data[1].T).T.contiguous()
    if kind in ("qr_lstsq", "qr_mixed"):
        a, b = data
        q, r = torch.linalg.qr(a)
        return torch.linalg.solve_triangular(r, (q.T @ b)[:, None], upper=True)[:, 0]
    # the textbook CG iteration, right-hand side by right-hand side block
    b = data[0]
    x = torch.zeros_like(b)
    for c in range(0, b.shape[0], 8):
        r = b[c: c + 8].clone()
        p, xs = r.clone(), x[c: c + 8]
        rr = (r * r).sum(1, keepdim=True)
        for _ in range(case["steps"]):
            ap = _poisson(p, case["nx"], case["ny"])
            alpha = rr / (p * ap).sum(1, keepdim=True)
            xs += alpha * p
            r -= alpha * ap
            new = (r * r).sum(1, keepdim=True)
            p = r + (new / rr) * p
            rr = new
    return x
