"""GPU: the FP32 QR's panels at the edges of their thread layout (one, two or
three rows per thread, 352 threads with rows, up to 16 CTAs) and of the panel
width, with the wide update running beside the next panel."""

import numpy as np
import pytest
import torch

from lineax_gb300 import mixed

pytestmark = pytest.mark.gpu


def q_of(h, tau):
    """Q's first n columns from LAPACK's raw factor (h: n × m, reflector j in
    row j), by applying the reflectors in FP64 to the identity."""
    n, m = h.shape
    q = torch.eye(m, n, dtype=torch.float64, device=h.device)
    for j in range(n - 1, -1, -1):
        v = h[j].clone()
        v[:j] = 0
        v[j] = 1
        q -= tau[j] * torch.outer(v, v @ q)
    return q


@pytest.mark.parametrize("m,n", [(4, 1), (4, 4), (64, 64), (68, 65), (352, 128), (356, 96),
                                 (2052, 129), (5632, 130), (5636, 64), (11264, 68), (11268, 132),
                                 (16896, 72), (16900, 66)])
def test_qr32_backward_error(dev, m, n):
    """A = Q R column by column: n reflections, each applied with products
    rounded to TF32 (2 x 2^-11 per product, random in sign over the m or 64
    terms of a sum) — 2^-10 sqrt(n) of the column's norm, twice that allowed."""
    a = np.random.default_rng(m + n).standard_normal((m, n))
    f = mixed.qr_factor_tf32(torch.tensor(a, device=dev))
    h, tau = f.h.double(), f.tau.double()
    q, r = q_of(h, tau), torch.triu(h[:, :n].t())
    err = torch.linalg.norm(torch.tensor(a, device=dev) - q @ r, dim=0)
    norm = torch.linalg.norm(torch.tensor(a, device=dev), dim=0)
    assert torch.all(err <= 2 * 2.0 ** -10 * n ** 0.5 * norm)


def test_qr32_zero_column(dev):
    """A zero column has the identity reflector (tau = 0)."""
    a = np.random.default_rng(0).standard_normal((400, 70))
    a[:, 0] = 0
    f = mixed.qr_factor_tf32(torch.tensor(a, device=dev))
    assert float(f.tau[0]) == 0.0 and torch.all(torch.isfinite(f.h))
