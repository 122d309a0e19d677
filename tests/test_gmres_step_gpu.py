"""GPU: one Arnoldi step of GMRES at the edges of its clusters (128 rows per CTA
before another is added, 16384 rows in all) and above them."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,restart", [(1, 2, 1), (2, 2, 2), (31, 3, 5), (127, 3, 5), (128, 3, 5),
                                         (129, 3, 5), (257, 2, 20), (300, 1, 128), (1025, 2, 9),
                                         (2049, 5, 4), (16384, 2, 6), (16385, 2, 6)])
def test_arnoldi_step_against_gram_schmidt(dev, n, k, restart):
    """V[j+1] = (w - V Vᵀw) / ||.|| with the device's own V: a dot of n terms errs
    by at most n 2^-53 ||w|| (unit V), the combination of j + 1 of them by
    (j + 1) times that and its own roundings; random w keeps ||.|| above half of
    ||w|| while j < n / 2."""
    lib = _ffi.load()
    nb = int(lib.lxgb_gmres_workspace_size(k, n, restart))
    buf = torch.zeros(nb // 8 + 64, dtype=torch.float64, device=dev)
    work = buf[(-buf.data_ptr() % 256) // 8:]
    st = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(n)
    r = torch.tensor(rng.standard_normal((k, n)), device=dev)
    on = torch.empty(k, dtype=torch.int32, device=dev)
    _ffi.call("lxgb_gmres_init", k, n, restart, _ffi.ptr(work), nb, st)
    _ffi.call("lxgb_gmres_cycle_begin", k, n, restart, 0, _ffi.ptr(r), _ffi.ptr(work), nb, st)

    def basis(j):
        off = int(lib.lxgb_gmres_basis_offset(k, n, restart, j)) // 8
        v = torch.as_strided(work, (k, n), ((restart + 1) * n, 1), work.storage_offset() + off)
        return v.cpu().numpy()

    vs = [basis(0)]
    for j in range(min(restart, max(1, n // 2))):
        w = rng.standard_normal((k, n))
        wd = torch.tensor(w, device=dev)
        _ffi.call("lxgb_gmres_arnoldi", k, n, restart, 0, j, _ffi.ptr(wd), _ffi.ptr(on),
                  _ffi.ptr(work), nb, st)
        assert torch.all(on == 1)
        got = basis(j + 1)
        for c in range(k):
            u = w[c] - sum(v[c] * (v[c] @ w[c]) for v in vs)
            if n == 1:  # nothing left: the step breaks down and divides by infinity
                assert np.all(got[c] == 0.0)
                continue
            ref = u / np.linalg.norm(u)
            scale = np.linalg.norm(w[c]) / np.linalg.norm(u)
            assert np.max(np.abs(got[c] - ref)) <= 4 * (j + 2) * n * 2.0 ** -53 * scale
        vs.append(got)


@pytest.mark.parametrize("n,k", [(130, 3), (300, 40), (5000, 9)])
def test_arnoldi_step_same_bits_beside_another_stream(dev, n, k):
    """The first step of a cycle (little work before the CTAs of a cluster exchange
    their sums) while another stream's products hold the SMs: the bits of the step
    made alone."""
    lib = _ffi.load()
    restart = 4
    nb = int(lib.lxgb_gmres_workspace_size(k, n, restart))
    buf = torch.zeros(nb // 8 + 64, dtype=torch.float64, device=dev)
    work = buf[(-buf.data_ptr() % 256) // 8:]
    st = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(n)
    r = torch.tensor(rng.standard_normal((k, n)), device=dev)
    w = torch.tensor(rng.standard_normal((k, n)), device=dev)
    on = torch.empty(k, dtype=torch.int32, device=dev)
    off = int(lib.lxgb_gmres_basis_offset(k, n, restart, 1)) // 8

    def step():
        _ffi.call("lxgb_gmres_init", k, n, restart, _ffi.ptr(work), nb, st)
        _ffi.call("lxgb_gmres_cycle_begin", k, n, restart, 0, _ffi.ptr(r), _ffi.ptr(work), nb, st)
        _ffi.call("lxgb_gmres_arnoldi", k, n, restart, 0, 0, _ffi.ptr(w.clone()), _ffi.ptr(on),
                  _ffi.ptr(work), nb, st)
        v = torch.as_strided(work, (k, n), ((restart + 1) * n, 1), work.storage_offset() + off)
        return v.clone()

    alone = step()
    g = torch.randn(6144, 6144, dtype=torch.bfloat16, device=dev)
    other = torch.cuda.Stream(dev)
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(other):
            for _ in range(4):
                g @ g
        assert torch.equal(step(), alone)
    torch.cuda.synchronize()
