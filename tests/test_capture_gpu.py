"""GPU: the multi-launch factorisations and solves under stream capture (they
use programmatic dependent launches, clusters and products beside a panel): a
replayed graph gives the bits of the direct calls, on new data too."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _dense, _ffi, mixed

pytestmark = pytest.mark.gpu


def lu(a, b):
    f, piv, info = _dense.lu_factor_batched(a)
    return [f, piv, info, _dense.lu_solve(f, piv, b), _dense.lu_solve(f, piv, b, trans=1)]


def cholesky(a, b):
    u = _dense.cho_factor(a @ a.T + a.shape[0] * torch.eye(a.shape[0], dtype=a.dtype, device=a.device))
    return [u, _dense.cho_solve(u, b)]


def qr(a, b):
    h, tau, t = _dense.geqrf(a)
    return [h, tau, _dense.ormqr(h, tau, t, b.reshape(1, -1).clone(), True)]


def fp32_factors(a, b):
    err = torch.zeros(1, dtype=torch.int32, device=a.device)
    f = mixed.lu_factor_tf32(a, "3xtf32", err=err)
    inv = mixed.lu_inverse(f, "3xtf32", err=err)
    q = mixed.qr_square_tf32(a, err=err)
    return [f.lu, f.piv, inv.linv, inv.uinv, inv.perm, q.qt, q.rinv, err]


def arnoldi(a, b):
    n, restart, lib = a.shape[0], 4, _ffi.load()
    nb = int(lib.lxgb_gmres_workspace_size(1, n, restart))
    buf = torch.zeros(nb // 8 + 64, dtype=torch.float64, device=a.device)
    work = buf[(-buf.data_ptr() % 256) // 8:]
    st = torch.cuda.current_stream().cuda_stream
    on = torch.empty(1, dtype=torch.int32, device=a.device)
    r = b.clone().reshape(1, -1)
    _ffi.call("lxgb_gmres_init", 1, n, restart, _ffi.ptr(work), nb, st)
    _ffi.call("lxgb_gmres_cycle_begin", 1, n, restart, 0, _ffi.ptr(r), _ffi.ptr(work), nb, st)
    out = []
    for j in range(restart):
        w = a[j].clone().reshape(1, -1)
        _ffi.call("lxgb_gmres_arnoldi", 1, n, restart, 0, j, _ffi.ptr(w), _ffi.ptr(on),
                  _ffi.ptr(work), nb, st)
        out.append(w)
    return out


@pytest.mark.parametrize("call", [lu, cholesky, qr, fp32_factors, arnoldi])
@pytest.mark.parametrize("n", [100, 324, 1200])
def test_replay_equals_direct_calls(dev, call, n):
    rng = np.random.default_rng(n)
    data = [(torch.tensor(rng.standard_normal((n, n)), device=dev),
             torch.tensor(rng.standard_normal(n), device=dev)) for _ in range(2)]
    direct = [[t.clone() for t in call(*d)] for d in data]
    a, b = data[0][0].clone(), data[0][1].clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(a, b)
    for (da, db), ref in zip(data, direct):
        a.copy_(da)
        b.copy_(db)
        graph.replay()
        torch.cuda.synchronize()
        for x, y in zip(out, ref):
            assert torch.equal(x, y)
