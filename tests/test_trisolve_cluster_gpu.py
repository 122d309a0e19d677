"""GPU: the one-launch triangular solve (a cluster per vector, up to four
vectors and 2048 unknowns) against the launch-per-block path on the same data:
the same bits for all flags, at the edges of blocks, clusters and of the rule."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lower,trans,unit", [(a, b, c) for a in (True, False)
                                              for b in (True, False) for c in (True, False)])
@pytest.mark.parametrize("n", [64, 65, 128, 129, 1000, 1024, 1025, 1089, 2048, 2049])
def test_cluster_equals_launch_per_block(dev, n, lower, trans, unit):
    g = torch.Generator(device=dev).manual_seed(n)
    t = torch.randn(n, n, dtype=torch.float64, device=dev, generator=g) / n
    t.diagonal().add_(1.0)
    b = torch.randn(40, n, dtype=torch.float64, device=dev, generator=g)
    many = _dense.trsv(t, b, lower=lower, trans=trans, unit=unit)
    for k in (1, 3, 4):
        assert torch.equal(_dense.trsv(t, b[:k], lower=lower, trans=trans, unit=unit), many[:k])
    m = torch.tril(t) if lower else torch.triu(t)
    if unit:
        m = m - torch.diag(m.diagonal()) + torch.eye(n, dtype=torch.float64, device=dev)
    m = m.t() if trans else m
    x = many[0]
    res = torch.abs(b[0] - m @ x)
    # (Higham 2002, theorem 8.5: |T - T'| <= gamma_n |T|, and the check's own product)
    assert torch.all(res <= (2 * n + 8) * 2.0 ** -53 * (torch.abs(m) @ torch.abs(x) + torch.abs(b[0])))


@pytest.mark.parametrize("n", [200, 1100])
@pytest.mark.parametrize("kind", ["tiny", "zero", "nan"])
def test_cluster_special_diagonals(dev, n, kind):
    """Entries whose scaling would underflow are divided in turn, zeros and NaN
    spread as in the other path."""
    g = torch.Generator(device=dev).manual_seed(n)
    t = torch.randn(n, n, dtype=torch.float64, device=dev, generator=g) / n
    t.diagonal().add_(1.0)
    i = n // 2
    if kind == "tiny":
        t *= 2.0 ** -1000
    else:
        t[i, i] = 0.0 if kind == "zero" else float("nan")
    b = torch.randn(40, n, dtype=torch.float64, device=dev, generator=g) * (2.0 ** -900 if kind == "tiny" else 1.0)
    many = _dense.trsv(t, b, lower=True, trans=False, unit=False)
    one = _dense.trsv(t, b[:1], lower=True, trans=False, unit=False)
    np.testing.assert_array_equal(one.cpu().numpy(), many[:1].cpu().numpy())
    assert bool(torch.isfinite(one).all()) == (kind == "tiny")
