"""GPU: the FP32 QR that also forms Q, with q right after h (shared products)
and elsewhere: the same bits, orthogonal Q, A = Q R."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _ffi, mixed

pytestmark = pytest.mark.gpu


def factor(a, joint):
    n, dev = a.shape[0], a.device
    lib = _ffi.load()
    if joint:
        h, q = torch.empty((2, n, n), dtype=torch.float32, device=dev)
    else:
        q, h = torch.empty((2, n, n), dtype=torch.float32, device=dev)
    tau = torch.empty(n, dtype=torch.float32, device=dev)
    t = torch.empty(int(lib.lxgb_geqrf_t_elems(n)), dtype=torch.float32, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    work = torch.empty(int(lib.lxgb_geqrf_f32_tc_q_workspace_size(n, n)) // 8 + 1,
                       dtype=torch.float64, device=dev)
    _ffi.call("lxgb_geqrf_f32_tc_q", n, n, _ffi.ptr(a), _ffi.ptr(h), _ffi.ptr(tau), _ffi.ptr(t),
              _ffi.ptr(q), _ffi.ptr(err), _ffi.ptr(work), work.numel() * 8,
              _ffi.stream_handle(dev))
    assert int(err.item()) == 0
    return h, q, tau


@pytest.mark.parametrize("n", [4, 60, 64, 68, 128, 132, 196, 520, 1028])
def test_qr32_q_joint_and_separate(dev, n):
    """Products rounded to TF32: columns of Q R within 2^-9 sqrt(n) of A's, Q
    orthogonal to the same."""
    a = torch.tensor(np.random.default_rng(n).standard_normal((n, n)), device=dev)
    h, q, tau = factor(a, True)
    h1, q1, tau1 = factor(a, False)
    assert torch.equal(torch.triu(h.t()), torch.triu(h1.t())) and torch.equal(tau, tau1)
    assert torch.equal(q, q1)
    qd, r = q.double(), torch.triu(h.double().t())
    tol = 2.0 ** -9 * n ** 0.5
    err = torch.linalg.norm(a - qd @ r, dim=0)
    assert torch.all(err <= tol * torch.linalg.norm(a, dim=0))
    eye = torch.eye(n, dtype=torch.float64, device=dev)
    assert torch.all(torch.linalg.norm(qd.t() @ qd - eye, dim=0) <= 2 * tol)


def test_qr_square_memory(dev):
    """The square QR's peak beside A: h and q, then R as rows beside them and the
    inversion's workspace (three matrices, not four); what stays is Qᵀ and R^{-1}."""
    n = 2048
    a = torch.tensor(np.random.default_rng(n).standard_normal((n, n)), device=dev)
    lib = _ffi.load()
    work = max(int(lib.lxgb_lu32_inverse_workspace_size(n, 1)),
               int(lib.lxgb_geqrf_f32_tc_q_workspace_size(n, n)))
    mixed.qr_square_tf32(a)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated(dev)
    torch.cuda.reset_peak_memory_stats(dev)
    qr = mixed.qr_square_tf32(a)
    small = 64 * n + 4 * 32 * n + (1 << 16)      # tau, T blocks, interchanges, rounding up
    assert torch.cuda.max_memory_allocated(dev) - before <= 12 * n * n + work + small
    assert torch.cuda.memory_allocated(dev) - before <= 8 * n * n + small
    x = torch.linalg.solve(a, torch.ones(n, dtype=torch.float64, device=dev))
    got = qr.rinv.double() @ (qr.qt.double() @ torch.ones(n, dtype=torch.float64, device=dev))
    # (TF32 products: a preconditioner's accuracy)
    assert torch.linalg.norm(got - x) <= 0.1 * torch.linalg.norm(x)
