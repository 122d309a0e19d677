"""GPU parity of the double-float block products at the edges of their tiles
(32 rows, 64 columns, 4 / 8 / 16 right-hand sides) and with rows that do not
start on 16-byte boundaries."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _ffi, mixed

pytestmark = pytest.mark.gpu


def _bound(n):
    """Relative to |A| |x|: both operands truncated to 2^-46, the lo x lo terms
    (at most 2^-46) left out, and FP32 roundings of the low-order sums, each
    2^-24 of at most an ulp (2^-24) per term."""
    return 3 * 2.0 ** -46 + n * 2.0 ** -48


def _work(nbytes, dev):
    return torch.empty(int(nbytes) // 8 + 1, dtype=torch.float64, device=dev)


@pytest.mark.parametrize("m,n,k", [(1, 1, 5), (31, 63, 5), (32, 64, 8), (33, 65, 9), (70, 130, 17),
                                   (129, 257, 16), (4160, 96, 7), (300, 1, 6)])
def test_full_products(dev, m, n, k):
    rng = np.random.default_rng(m * n + k)
    a, x, b = rng.standard_normal((m, n)), rng.standard_normal((k, n)), rng.standard_normal((k, m))
    sp = mixed.split_matrix(torch.tensor(a, device=dev))
    xt, bt = torch.tensor(x, device=dev), torch.tensor(b, device=dev)
    y = torch.empty((k, m), dtype=torch.float64, device=dev)
    work = _work(_ffi.load().lxgb_gemv_df_workspace_size(n, k), dev)
    scale = np.abs(x) @ np.abs(a).T
    for lo in (sp.lo, None):
        mat = a if lo is not None else sp.hi.double().cpu().numpy()
        for bb in (None, bt):
            _ffi.call("lxgb_gemv_df", m, n, _ffi.ptr(sp.hi), _ffi.ptr(lo), n, k, _ffi.ptr(xt), n,
                      _ffi.ptr(bb), _ffi.ptr(y), m, 1, _ffi.ptr(work), work.numel() * 8,
                      _ffi.stream_handle(dev))
            ref = x @ mat.T if bb is None else b - x @ mat.T
            err = np.abs(y.cpu().numpy() - ref)
            assert (err <= _bound(n) * scale + n * 2.0 ** -53 * scale).all()


@pytest.mark.parametrize("n,k", [(1, 1), (31, 2), (64, 16), (70, 5), (100, 20), (513, 3)])
def test_triangular_products(dev, n, k):
    """lxgb_lu32_apply with given triangles (zeros in the other half)."""
    rng = np.random.default_rng(n + k)
    low = np.tril(rng.standard_normal((n, n))).astype(np.float32)
    up = np.triu(rng.standard_normal((n, n))).astype(np.float32)
    perm = rng.permutation(n).astype(np.int32)
    x = rng.standard_normal((k, n))
    inv = mixed.InverseLU32(torch.tensor(low, device=dev), torch.tensor(up, device=dev),
                            torch.tensor(perm, device=dev))
    y = mixed.InverseLUPreconditioner(None, inv, "df").mv_block(torch.tensor(x, device=dev))
    l64, u64 = low.astype(np.float64), up.astype(np.float64)
    ref = (u64 @ (l64 @ x[:, perm].T)).T
    scale = (np.abs(u64) @ (np.abs(l64) @ np.abs(x[:, perm]).T)).T
    assert (np.abs(y.cpu().numpy() - ref) <= 3 * _bound(n) * scale).all()
