"""GPU parity of the blocked FP64 LU (n > 168) at the edges of its panel
kernel: one to sixteen CTAs per panel, four, two and one threads per row."""

import numpy as np
import pytest
import scipy.linalg as sl
import torch

from lineax_gb300 import _dense
from oracle.build import getf2_batched

pytestmark = pytest.mark.gpu


def _matrix(n):
    rng = np.random.default_rng(n)
    return rng.standard_normal((n, n)) / np.sqrt(n) + np.eye(n)


@pytest.mark.parametrize("n", [170, 513, 545, 1000, 2081])
def test_blocked_lu_bit_exact_vs_getf2_twin(dev, n):
    """Bit for bit the getf2 recurrence (2081: its first panels have two
    threads per row)."""
    a = _matrix(n)
    lu, piv, info = _dense.lu_factor_batched(torch.tensor(a[None], device=dev))
    lu_ref, piv_ref, info_ref = getf2_batched(a[None])
    np.testing.assert_array_equal(piv.cpu().numpy(), piv_ref)
    np.testing.assert_array_equal(info.cpu().numpy(), info_ref)
    assert np.array_equal(lu.cpu().numpy(), lu_ref)


def test_blocked_lu_one_thread_per_row(dev):
    """First panels with one thread per row (n > 4096): LAPACK's pivots, and
    |P A - L U| <= n u / (1 - n u) |L| |U| (the factorisation's own bound;
    twice that for the products formed here)."""
    n = 4130
    a = torch.tensor(_matrix(n), device=dev)
    lu, piv = _dense.lu_factor(a)
    ref_lu, ref_piv = sl.lu_factor(a.cpu().numpy(), check_finite=False)
    np.testing.assert_array_equal(piv.cpu().numpy(), ref_piv)
    perm = np.arange(n)
    for k, p in enumerate(ref_piv):
        perm[[k, p]] = perm[[p, k]]
    low = torch.tril(lu, -1) + torch.eye(n, dtype=torch.float64, device=dev)
    up = torch.triu(lu)
    err = (a[torch.tensor(perm, device=dev)] - low @ up).abs()
    bound = 2 * n * 2.0 ** -53 * (low.abs() @ up.abs())
    assert bool((err <= bound).all())


def test_blocked_lu_zero_and_nan_columns(dev):
    """A zero column inside a later panel (info, no interchange) and a column
    of NaNs, against the twin."""
    for kind in ("zero", "nan"):
        a = _matrix(300)
        a[:, 100] = 0.0 if kind == "zero" else np.nan
        lu, piv, info = _dense.lu_factor_batched(torch.tensor(a[None], device=dev))
        lu_ref, piv_ref, info_ref = getf2_batched(a[None])
        np.testing.assert_array_equal(piv.cpu().numpy(), piv_ref)
        np.testing.assert_array_equal(info.cpu().numpy(), info_ref)
        np.testing.assert_array_equal(lu.cpu().numpy(), lu_ref)
