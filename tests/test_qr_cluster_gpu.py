"""GPU checks of the cluster Householder QR at the edges of its 16- and
32-column blocks, its rows per CTA and the largest panel (8192 rows)."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _dense

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("m,n", [(2, 2), (16, 16), (17, 16), (33, 17), (64, 33), (200, 48),
                                 (65, 65), (513, 49), (1025, 40), (2049, 33), (4100, 18),
                                 (8192, 35), (8193, 18)])
def test_q_transposed_a_is_r(dev, m, n):
    """Qᵀ A = [R; 0] and Q (Qᵀ c) = c, with Q applied panel by panel: column
    errors at most 20 n u ||a_j|| (n reflectors, each within a few u)."""
    rng = np.random.default_rng(m + n)
    a = torch.tensor(rng.standard_normal((m, n)), device=dev)
    h, tau, t = _dense.geqrf(a)
    qta = _dense.ormqr(h, tau, t, a.T.contiguous(), trans=True)      # rows: Qᵀ a_j
    r = torch.triu(h[:, :n].T)                                       # R[i][j] = h[j][i]
    want = torch.zeros(n, m, dtype=torch.float64, device=dev)
    want[:, :n] = r.T
    norms = a.norm(dim=0)
    assert bool(((qta - want).norm(dim=1) <= 20 * n * U * norms).all())
    c = torch.tensor(rng.standard_normal((3, m)), device=dev)
    back = _dense.ormqr(h, tau, t, _dense.ormqr(h, tau, t, c, trans=True), trans=False)
    assert bool(((back - c).norm(dim=1) <= 40 * n * U * c.norm(dim=1)).all())
    # tau of unit-leading reflectors: tau ||v||² = 2
    v = torch.tril(h.T, -1)
    v[torch.arange(n), torch.arange(n)] = 1.0
    live = tau != 0
    assert bool(((tau * (v * v).sum(0) - 2).abs()[live] <= 100 * U).all())


def test_qr_zero_columns_and_extreme_scales(dev):
    """A zero column (tau = 0, nothing changed) and columns whose squares
    overflow or underflow next to the others (the hypot path)."""
    rng = np.random.default_rng(1)
    a = rng.standard_normal((300, 40))
    a[:, 7] = 0.0
    scale = np.ones(40)
    scale[20:] = 1e140
    a = torch.tensor(a * scale, device=dev)
    h, tau, t = _dense.geqrf(a)
    assert bool(torch.isfinite(h).all())
    qta = _dense.ormqr(h, tau, t, a.T.contiguous(), trans=True)
    r = torch.triu(h[:, :40].T)
    err = (qta[:, :40].T - r).abs().amax(0)
    assert bool((err <= 20 * 40 * U * a.norm(dim=0)).all())


@pytest.mark.parametrize("m,n", [(300, 40), (3001, 33)])
@pytest.mark.parametrize("scale", [1e-150, 1e-130, 1e-100, 1e100, 1e150])
def test_qr_columns_outside_the_reciprocal_root_range(dev, m, n, scale):
    """Squared norms below and above the exponents for which a reflector is formed from
    a reciprocal root (2^-823 and 2^877, a leading entry above 2^477): the error bound
    of test_q_transposed_a_is_r, for those columns and their neighbours.  (300 squares of
    1e-150 are normal numbers and of 1e150 finite.)"""
    rng = np.random.default_rng(m)
    a = rng.standard_normal((m, n))
    a[:, 3:6] *= scale
    a[:, n // 2:] *= scale
    a = torch.tensor(a, device=dev)
    h, tau, t = _dense.geqrf(a)
    qta = _dense.ormqr(h, tau, t, a.T.contiguous(), trans=True)
    want = torch.zeros(n, m, dtype=torch.float64, device=dev)
    want[:, :n] = torch.triu(h[:, :n].T).T
    err = ((qta - want) / scale).norm(dim=1) * scale if scale < 1 else (qta - want).norm(dim=1)
    assert bool((err <= 20 * n * U * a.norm(dim=0)).all())
    v = torch.tril(h.T, -1)
    v[torch.arange(n), torch.arange(n)] = 1.0
    assert bool(((tau * (v * v).sum(0) - 2).abs() <= 100 * U).all())


@pytest.mark.parametrize("m,n", [(300, 40), (1025, 33), (2000, 100), (4100, 18), (8192, 35)])
@pytest.mark.parametrize("k", [100, 300, 650])
def test_q_of_many_vectors(dev, m, n, k):
    """Many vectors at once, with fewer CTAs for each: within the bound of
    test_q_transposed_a_is_r of the vectors taken three at a time, and back."""
    g = torch.Generator(device=dev).manual_seed(k)
    h, tau, t = _dense.geqrf(torch.randn(m, n, dtype=torch.float64, device=dev, generator=g))
    c = torch.randn(k, m, dtype=torch.float64, device=dev, generator=g)
    some = list(range(0, k, 37))
    for trans in (True, False):
        y = _dense.ormqr(h, tau, t, c, trans=trans)
        for i in range(0, len(some), 3):
            s = some[i:i + 3]
            few = _dense.ormqr(h, tau, t, c[s].contiguous(), trans=trans)
            assert bool(((y[s] - few).norm(dim=1) <= 40 * n * U * c[s].norm(dim=1)).all())
        back = _dense.ormqr(h, tau, t, y, trans=not trans)
        assert bool(((back - c).norm(dim=1) <= 40 * n * U * c.norm(dim=1)).all())


@pytest.mark.parametrize("m,n,k", [(5, 3, 1), (40, 16, 5), (300, 16, 0), (300, 16, 15), (700, 12, 7)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_qr_non_finite_column_leaves_finished_rows_alone(dev, m, n, k, bad):
    """Column k with a non-finite entry in the last row: the columns before it, and the
    rows of R that the reflectors before k made, keep the bits they have without it."""
    rng = np.random.default_rng(m + n)
    a = torch.tensor(rng.standard_normal((m, n)), device=dev)
    h0, tau0, _ = _dense.geqrf(a)
    a[m - 1, k] = bad
    h, tau, _ = _dense.geqrf(a)
    assert torch.equal(h[:k], h0[:k]) and torch.equal(tau[:k], tau0[:k])
    assert torch.equal(h[k + 1:, :k], h0[k + 1:, :k])
