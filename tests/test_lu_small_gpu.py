"""GPU: the one-CTA LU and its solve at the edges of their blocks (16 and 32
unknowns, 64 and 128 rows), with several right-hand sides, zero and NaN pivots."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _dense

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def getf2(a):
    """LAPACK's unblocked recurrence in the engine's arithmetic but for the FMAs'
    single rounding: pivots (first row of max |a|)."""
    a, piv = a.copy(), []
    n = a.shape[0]
    for k in range(n):
        p = k + int(np.argmax(np.abs(a[k:, k])))
        piv.append(p)
        a[[k, p]] = a[[p, k]]
        a[k + 1:, k] /= a[k, k]
        a[k + 1:, k + 1:] -= np.outer(a[k + 1:, k], a[k, k + 1:])
    return a, piv


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 97, 127, 128, 129, 160,
                               161, 167, 168])
@pytest.mark.parametrize("batch,nrhs", [(1, 1), (3, 2), (2, 4), (1, 9)])
def test_lu_small_factor_and_solve(dev, n, batch, nrhs):
    """|P A - L U| <= n u |L| |U| and |b - A x| <= 3 n u |A-ish| |x| (Higham 2002,
    theorems 9.3 and 9.4, gamma_n <= 1.01 n u); the unknowns of U are multiplied
    by the rounded inverse of the diagonal: one more rounding each."""
    rng = np.random.default_rng(n + batch)
    a = rng.standard_normal((batch, n, n))
    b = rng.standard_normal((batch, nrhs, n))
    lu_d, piv_d, info = _dense.lu_factor_batched(torch.tensor(a, device=dev))
    assert torch.all(info == 0)
    x = _dense.lu_solve_batched(lu_d, piv_d, torch.tensor(b, device=dev)).cpu().numpy()
    xt = _dense.lu_solve_batched(lu_d, piv_d, torch.tensor(b, device=dev), trans=1).cpu().numpy()
    lu, piv = lu_d.cpu().numpy(), piv_d.cpu().numpy()
    for s in range(batch):
        assert list(piv[s]) == getf2(a[s])[1]
        l, u = np.tril(lu[s], -1) + np.eye(n), np.triu(lu[s])
        perm = np.arange(n)
        for k, p in enumerate(piv[s]):
            perm[[k, p]] = perm[[p, k]]
        mod = np.abs(l) @ np.abs(u)
        assert np.all(np.abs(a[s][perm] - l @ u) <= (n + 2) * U * mod)
        back = np.empty((n, n))
        back[perm] = mod
        for c in range(nrhs):
            res = np.abs(b[s, c] - a[s] @ x[s, c])
            assert np.all(res <= (3 * n + 8) * U * (back @ np.abs(x[s, c])))
            res = np.abs(b[s, c] - a[s].T @ xt[s, c])
            assert np.all(res <= (3 * n + 8) * U * (back.T @ np.abs(xt[s, c])))


@pytest.mark.parametrize("n,col", [(5, 0), (40, 31), (64, 63), (100, 64), (168, 167)])
def test_lu_small_zero_and_nan_columns(dev, n, col):
    """A zero column: info names it and every other step goes on; a column of
    NaNs keeps its row (NaN is never chosen)."""
    a = np.random.default_rng(col).standard_normal((n, n))
    a[:, col] = 0
    _, piv, info = _dense.lu_factor_batched(torch.tensor(a, device=dev))
    assert int(info) == col + 1 and int(piv[col]) == col
    a[:, col] = np.nan
    lu, piv, info = _dense.lu_factor_batched(torch.tensor(a, device=dev))
    assert int(info) == 0 and int(piv[col]) == col
    assert torch.all(torch.isnan(lu[col:, col]))


@pytest.mark.parametrize("n", [20, 100])
def test_lu_small_tiny_pivots_divide(dev, n):
    """Pivots below DBL_MIN (their reciprocal overflows): the multipliers are
    quotients."""
    a = np.tril(np.random.default_rng(n).uniform(0.25, 0.5, (n, n)), -1) + np.eye(n)
    s = np.ldexp(1.0, -1060)
    lu, piv, info = _dense.lu_factor_batched(torch.tensor(a * s, device=dev))
    assert int(info) == 0 and list(piv.cpu().numpy()) == list(range(n))
    ref = np.tril(a * s, -1) / s
    assert np.array_equal(np.tril(lu.cpu().numpy(), -1), ref)


@pytest.mark.parametrize("n", [64, 65, 80, 81, 96, 119, 120, 168])
def test_lu_small_large_batches_same_bits(dev, n):
    """More matrices than SMs, and than two per SM: fewer threads per matrix where an SM
    holds several, the bits of the matrix factored alone."""
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    g = torch.Generator(device=dev).manual_seed(n)
    a = torch.randn(2 * sms + 1, n, n, dtype=torch.float64, device=dev, generator=g)
    one = [_dense.lu_factor_batched(a[s:s + 1]) for s in range(0, 2 * sms + 1, 37)]
    for batch in (sms + 1, 2 * sms + 1):
        lu, piv, info = _dense.lu_factor_batched(a[:batch])
        assert torch.all(info == 0)
        for i, s in enumerate(range(0, batch, 37)):
            assert torch.equal(lu[s], one[i][0][0]) and torch.equal(piv[s], one[i][1][0])


def test_lu_small_time_of_large_batches(dev):
    """A matrix of order 65 in a batch of 4096 takes little more than one of order 64
    (65^3 / 64^3 = 1.05, and one more block of rows): not half as long again."""
    def us(n):
        g = torch.Generator(device=dev).manual_seed(n)
        a = torch.randn(4096, n, n, dtype=torch.float64, device=dev, generator=g)
        best = np.inf
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            _dense.lu_factor_batched(a)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert us(65) <= 1.5 * us(64)


@pytest.mark.parametrize("n", [1, 16, 31, 32, 33, 64, 65, 128, 168])
@pytest.mark.parametrize("nrhs", [5, 8, 9, 17])
def test_lu_small_solve_same_bits_one_by_one(dev, n, nrhs):
    """More than four right-hand sides go two to a warp: the bits of each alone."""
    g = torch.Generator(device=dev).manual_seed(n)
    a = torch.randn(2, n, n, dtype=torch.float64, device=dev, generator=g)
    b = torch.randn(2, nrhs, n, dtype=torch.float64, device=dev, generator=g)
    lu, piv, _ = _dense.lu_factor_batched(a)
    for trans in (0, 1):
        x = _dense.lu_solve_batched(lu, piv, b, trans)
        for c in range(nrhs):
            assert torch.equal(x[:, c], _dense.lu_solve_batched(lu, piv, b[:, c].contiguous(), trans))
