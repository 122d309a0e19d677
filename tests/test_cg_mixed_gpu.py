"""GPU: the passes of the mixed-precision Poisson CG at the edges of their tiles
(256 columns, 16 rows, 16-byte rows or not, one or many partial sums per CTA)."""

import numpy as np
import pytest
import torch

import lineax_gb300 as lx
from lineax_gb300 import _krylov

pytestmark = pytest.mark.gpu


def poisson(v):
    out = 4.0 * v
    out[1:] -= v[:-1]
    out[:-1] -= v[1:]
    out[:, 1:] -= v[:, :-1]
    out[:, :-1] -= v[:, 1:]
    return out


def cg(b, steps):
    """`steps` iterations of CG from zero in FP64."""
    x, r = np.zeros_like(b), b.copy()
    p, g = r.copy(), np.sum(b * b)
    for _ in range(steps):
        q = poisson(p)
        al = g / np.sum(p * q)
        x += al * p
        r -= al * q
        g, g0 = np.sum(r * r), g
        p = r + (g / g0) * p
    return x


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 300), (300, 1), (16, 256), (17, 257), (15, 255),
                                   (33, 260), (50, 1001), (128, 512), (301, 252)])
@pytest.mark.parametrize("steps", [1, 2, 7])
def test_cg_mixed_steps_against_fp64(dev, nx, ny, steps):
    """x after a few steps: the FP32 vectors carry about 20 roundings of 2^-24
    per step, a few of them summed up by alpha and beta: 1e-4 of max |x| is two
    orders above 7 x 20 x 2^-24."""
    steps = min(steps, nx * ny)
    k = 3
    b = np.random.default_rng(nx * ny).standard_normal((k, nx, ny))
    op = lx.Poisson2DOperator(nx, ny)
    res = _krylov.cg_poisson_mixed(op, torch.tensor(b.reshape(k, -1), device=dev), rtol=1e-14,
                                   atol=1e-14, max_steps=steps)
    x = res.y.cpu().numpy().reshape(k, nx, ny)
    for c in range(k):
        ref = cg(b[c], steps)
        assert np.max(np.abs(x[c] - ref)) <= 1e-4 * np.max(np.abs(ref))


@pytest.mark.parametrize("nx,ny", [(300, 252), (299, 253), (64, 1030)])
def test_cg_mixed_same_alone_and_in_a_block(dev, nx, ny):
    """The number of right-hand sides chooses how many partial sums a CTA forms;
    every right-hand side has the same bits whichever it is."""
    b = torch.randn(400, nx * ny, dtype=torch.float64, device=dev,
                    generator=torch.Generator(device=dev).manual_seed(ny))
    op = lx.Poisson2DOperator(nx, ny)
    run = lambda v: _krylov.cg_poisson_mixed(op, v, rtol=1e-10, atol=1e-10, max_steps=20).y
    block = run(b)
    for c, k in ((0, 1), (7, 40), (399, 1)):
        assert torch.equal(run(b[c:c + k]), block[c:c + k])
