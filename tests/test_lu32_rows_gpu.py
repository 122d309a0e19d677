"""GPU: the FP32 LU's panels and block rows at the edges of their tiles (64
columns, one row per thread of 512) and with interchanges of every kind:
inside the panel, outside it, several with the same outside row."""

import numpy as np
import pytest
import torch

from lineax_gb300 import mixed

pytestmark = pytest.mark.gpu


def swaps_to_perm(piv):
    perm = np.arange(len(piv))
    for k, p in enumerate(piv):
        perm[[k, p]] = perm[[p, k]]
    return perm


@pytest.mark.parametrize("precision,ulp", [("tf32", 2.0 ** -10), ("3xtf32", 2.0 ** -21),
                                           ("bf16", 2.0 ** -7)])
@pytest.mark.parametrize("n", [4, 60, 64, 68, 128, 508, 512, 516, 1100])
def test_lu32_componentwise_residual(dev, n, precision, ulp):
    """|P A - L U| <= n u |L| |U| componentwise (Higham 2002, theorem 9.3), u the
    rounding of a product: operands rounded to TF32 or BF16 (2 x 2^-11, 2 x 2^-8),
    about 2^-22 with 3xTF32 — twice that allowed."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    f = mixed.lu_factor_tf32(torch.tensor(a, device=dev), precision)
    assert int(f.info) == 0
    lu = f.lu.double().cpu().numpy()
    l, u = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    err = np.abs(a[swaps_to_perm(f.piv.cpu().numpy())] - l @ u)
    assert np.all(err <= n * ulp * (np.abs(l) @ np.abs(u)))


@pytest.mark.parametrize("n", [64, 68, 200, 516])
@pytest.mark.parametrize("order", ["cycle", "cycle_back", "reverse", "far", "random"])
def test_lu32_interchanges_exact(dev, n, order):
    """A permuted diagonal matrix: every pivot is forced, L = I and U is the
    diagonal, exactly.  'far' sends the rows of a panel to the last rows."""
    perm = {"cycle": np.roll(np.arange(n), 1), "cycle_back": np.roll(np.arange(n), -1),
            "reverse": np.arange(n)[::-1], "far": np.roll(np.arange(n), n // 2),
            "random": np.random.default_rng(n).permutation(n)}[order]
    d = np.arange(1, n + 1, dtype=np.float64)
    a = np.diag(d)[perm]
    f = mixed.lu_factor_tf32(torch.tensor(a, device=dev), "3xtf32")
    assert np.array_equal(f.lu.cpu().numpy(), np.diag(d).astype(np.float32))
    assert np.array_equal(a[swaps_to_perm(f.piv.cpu().numpy())], np.diag(d))
    inv = mixed.lu_inverse(f, "3xtf32")
    assert np.array_equal(inv.linv.cpu().numpy(), np.eye(n, dtype=np.float32))
    assert np.array_equal(inv.uinv.cpu().numpy(), np.diag(np.float32(1) / d.astype(np.float32)))
    assert np.array_equal(inv.perm.cpu().numpy(), swaps_to_perm(f.piv.cpu().numpy()))


@pytest.mark.parametrize("n,col", [(64, 0), (200, 63), (200, 70), (200, 199)])
def test_lu32_zero_column_is_reported(dev, n, col):
    """A zero column stays zero through the updates: info names it (1-based)."""
    a = np.random.default_rng(col).standard_normal((n, n))
    a[:, col] = 0
    f = mixed.lu_factor_tf32(torch.tensor(a, device=dev), "3xtf32")
    assert int(f.info) == col + 1
