"""GPU parity of the multi-CTA triangular solve and of the LU solve's row
interchanges, at the edges of their 32- and 64-unknown blocks."""

import numpy as np
import pytest
import torch

from lineax_gb300 import _dense, _ffi

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _t(x, dev):
    return torch.tensor(np.asarray(x), dtype=torch.float64, device=dev)


@pytest.mark.parametrize("lower,trans", [(True, False), (False, False), (True, True),
                                         (False, True)])
@pytest.mark.parametrize("n", [1, 32, 33, 63, 64, 65, 96, 97, 129, 200])
def test_trsm_block_edges(dev, n, lower, trans):
    """Componentwise backward error of substitution with rounded reciprocals:
    |op(T) x - b| <= (n + 4) u |op(T)| |x| (residual in extended precision),
    for three vectors and rows longer than the matrix."""
    rng = np.random.default_rng(n)
    m = rng.standard_normal((n, n + 5))
    m[np.arange(n), np.arange(n)] += np.sign(m[np.arange(n), np.arange(n)])
    b = rng.standard_normal((3, n))
    x = _dense.trsv(_t(m, dev)[:, :n] if n == 1 else _t(m, dev), _t(b, dev), lower=lower,
                    trans=trans, unit=False).cpu().numpy()
    tri = np.tril(m[:, :n]) if lower else np.triu(m[:, :n])
    tri = tri.T if trans else tri
    for c in range(3):
        res = np.abs(tri.astype(np.longdouble) @ x[c].astype(np.longdouble) - b[c])
        assert (res <= (n + 4) * U * (np.abs(tri) @ np.abs(x[c]))).all()


@pytest.mark.parametrize("scale", [1e-250, 1e250])
def test_trsm_extreme_scaling_divides(dev, scale):
    """Entries too large or small to be scaled ahead take the dividing path:
    the backward error bound of test_trsm_block_edges."""
    n = 70
    rng = np.random.default_rng(3)
    m = np.tril(np.sign(rng.standard_normal((n, n))) * 2.0 ** rng.integers(-2, 3, (n, n)))
    m[40:, :] *= scale
    m[np.arange(n), np.arange(n)] = np.where(np.arange(n) < 40, 1.0, scale)
    b = m.sum(1)
    x = _dense.trsv(_t(m, dev), _t(b, dev), lower=True, trans=False, unit=False).cpu().numpy()
    res = np.abs(m.astype(np.longdouble) @ x.astype(np.longdouble) - b)
    assert (res <= (n + 4) * U * (np.abs(m) @ np.abs(x))).all()


def test_trsm_zero_diagonal_is_not_finite(dev):
    m = np.eye(100)
    m[70, 70] = 0.0
    x = _dense.trsv(_t(m, dev), _t(np.ones(100), dev), lower=True, trans=False,
                    unit=False).cpu().numpy()
    assert np.isinf(x[70]) and np.isfinite(x[:70]).all()


@pytest.mark.parametrize("n", [169, 300, 1200])
@pytest.mark.parametrize("kind", ["random", "shift", "last", "none", "any"])
def test_getrs_interchanges(dev, n, kind):
    """P b and Pᵀ b of pivot sequences with long and short chains (and of one
    with partners above the diagonal), through identity factors: exact."""
    rng = np.random.default_rng(n)
    k = np.arange(n)
    piv = {"random": k + (rng.random(n) * (n - k)).astype(int), "shift": np.minimum(k + 1, n - 1),
           "last": np.full(n, n - 1), "none": k, "any": rng.integers(0, n, n)}[kind]
    b = rng.standard_normal((2, 3, n))
    lu = _t(np.stack([np.eye(n)] * 2), dev)
    pv = torch.tensor(np.stack([piv] * 2).astype(np.int32), device=dev)
    for trans in (0, 1):
        ref = b.copy()
        for i in (range(n) if not trans else range(n - 1, -1, -1)):
            ref[..., [i, piv[i]]] = ref[..., [piv[i], i]]
        got = _dense.lu_solve_batched(lu, pv, _t(b, dev), trans=trans).cpu().numpy()
        np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("lower,trans", [(True, False), (False, False), (True, True),
                                         (False, True)])
@pytest.mark.parametrize("unit", [False, True])
@pytest.mark.parametrize("n", [40, 65, 300, 2100])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_trsm_non_finite_right_hand_side(dev, n, lower, trans, unit, bad):
    """A non-finite b_k with finite, well-scaled entries: the unknowns solved before
    it have the bits of the finite solve, x_k is b_k (a positive diagonal keeps its
    sign), those after it are not finite.  One vector, and as many as take the other
    path."""
    rng = np.random.default_rng(n)
    m = _t(rng.uniform(0.5, 1.0, (n, n)) / n, dev)
    m.diagonal().add_(1.0)
    b = rng.standard_normal(n)
    order = np.arange(n) if lower != trans else np.arange(n)[::-1]
    for k in (0, 7, n // 2, n - 1):
        b2 = b.copy()
        b2[order[k]] = bad
        for nv in (1, 40):
            args = dict(lower=lower, trans=trans, unit=unit)
            good = _dense.trsv(m, _t(np.tile(b, (nv, 1)), dev), **args).cpu().numpy()
            x = _dense.trsv(m, _t(np.tile(b2, (nv, 1)), dev), **args).cpu().numpy()
            np.testing.assert_array_equal(x[:, order[:k]], good[:, order[:k]])
            np.testing.assert_array_equal(x[:, order[k]], np.full(nv, bad))
            assert not np.isfinite(x[:, order[k + 1:]]).any()


@pytest.mark.parametrize("n", [1, 40, 65, 300, 2100])
@pytest.mark.parametrize("lower", [True, False])
def test_trsm_diagonal_matrix_is_correctly_rounded(dev, n, lower):
    """With a diagonal T each unknown is one quotient, rounded once: the bits of
    b / t, for three vectors and for as many as take the other path."""
    rng = np.random.default_rng(n)
    d = rng.uniform(1.0, 100.0, n).round(1)
    b = rng.standard_normal((40, n))
    b[0] = d                                     # x = 1
    b[1] = np.resize([0.0, -0.0, 5e-324, -1e-310, 1e300, -1.7e308, 3e-200, 7e180], n)
    b[2] = -0.0
    for nv in (3, 40):
        x = _dense.trsv(_t(np.diag(d), dev), _t(b[:nv], dev), lower=lower, trans=False,
                        unit=False).cpu().numpy()
        np.testing.assert_array_equal(x, b[:nv] / d)
        # (the zeros of T turn the sign of a zero after the first unknown)
        assert np.signbit(x[2, 0 if lower else n - 1])


def _partners(kind, n, rng):
    k = np.arange(n)
    return {"random": k + (rng.random(n) * (n - k)).astype(int), "shift": np.minimum(k + 1, n - 1),
            "last": np.full(n, n - 1), "halves": np.where(k < n // 2, n // 2 + k % 3, n - 1 - k % 2),
            "any": rng.integers(0, n, n), "none": k}[kind].astype(np.int32)


def _interchanged(b, piv, trans):
    ref = b.copy()
    for i in (range(len(piv)) if not trans else range(len(piv) - 1, -1, -1)):
        if piv[i] != i:
            ref[..., [i, piv[i]]] = ref[..., [piv[i], i]]
    return ref


@pytest.mark.parametrize("n", [1001, 11000, 11001, 19200, 19201])
@pytest.mark.parametrize("kind", ["random", "shift", "last", "halves", "any"])
def test_getrs_interchanges_long_lists_and_large_orders(dev, n, kind):
    """The interchanges at the ends of the ranges of the one-gather path, with lists of
    one partner longer than a row walks (they are then ordered by one warp) and with
    chains of n links: exact, through identity factors."""
    rng = np.random.default_rng(n)
    piv = np.maximum(_partners(kind, n, rng), np.arange(n) if kind != "any" else 0).astype(np.int32)
    b = rng.standard_normal((2, n))
    lu = torch.eye(n, dtype=torch.float64, device=dev)
    for trans in (0, 1):
        got = _dense.lu_solve_batched(lu[None], torch.tensor(piv[None], device=dev), _t(b[None], dev),
                                      trans=trans).cpu().numpy()[0]
        np.testing.assert_array_equal(got, _interchanged(b, piv, trans))


@pytest.mark.parametrize("n", [64, 1028, 8192, 20000])
@pytest.mark.parametrize("kind", ["random", "shift", "last", "halves", "any"])
def test_lu32_interchanges_as_one_gather(dev, n, kind):
    """The gather that lxgb_lu32_inverse returns, for the same sequences."""
    rng = np.random.default_rng(n)
    piv = np.maximum(_partners(kind, n, rng), np.arange(n) if kind != "any" else 0).astype(np.int32)
    lib = _ffi.load()
    lu, linv = (torch.eye(n, dtype=torch.float32, device=dev) for _ in range(2))
    perm = torch.empty(n, dtype=torch.int32, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    nb = int(lib.lxgb_lu32_inverse_workspace_size(n, 0))
    work = torch.empty(nb // 8 + 1, dtype=torch.float64, device=dev)
    pv = torch.tensor(piv, device=dev)
    _ffi.call("lxgb_lu32_inverse", n, _ffi.ptr(lu), _ffi.ptr(pv), _ffi.ptr(linv), None,
              _ffi.ptr(perm), 0, _ffi.ptr(err), _ffi.ptr(work), nb,
              torch.cuda.current_stream().cuda_stream)
    np.testing.assert_array_equal(perm.cpu().numpy(), _interchanged(np.arange(n), piv, 0))


def _solve_ms(dev, n, kind):
    lu = torch.eye(n, dtype=torch.float64, device=dev)
    b = torch.ones(1, 1, n, dtype=torch.float64, device=dev)
    piv = torch.tensor(_partners(kind, n, np.random.default_rng(0))[None], device=dev)
    best = np.inf
    for _ in range(6):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        _dense.lu_solve_batched(lu[None], piv, b, trans=0)
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def test_getrs_interchanges_time_does_not_grow_with_the_list(dev):
    """All rows with one partner, and a cyclic shift: the solve takes no longer than
    without interchanges by more than a quarter (walking every list from every row it
    took 1.3 times as long and more; a row walks at most 64 links)."""
    none = _solve_ms(dev, 11000, "none")
    for kind in ("last", "shift", "random"):
        assert _solve_ms(dev, 11000, kind) <= 1.25 * none


def test_getrs_interchanges_time_of_large_orders(dev):
    """Orders above 11000 take the same path: per unknown no more than a quarter above
    n = 11000 (one thread exchanging in memory took 1.5 ms of a solve of 3)."""
    assert _solve_ms(dev, 13000, "random") <= 1.25 * 13000 / 11000 * _solve_ms(dev, 11000, "random")


@pytest.mark.parametrize("lower,trans,unit", [(a, b, c) for a in (True, False)
                                              for b in (True, False) for c in (True, False)])
@pytest.mark.parametrize("n", [1, 32, 33, 64, 65, 96, 97, 129, 1000, 4096, 4097])
def test_trsm_many_vectors_same_bits_as_some(dev, n, lower, trans, unit):
    """The vectors that one launch takes together (from one and a half per SM on, and two
    per CTA above four or eight) against the same vectors 40 at a time."""
    g = torch.Generator(device=dev).manual_seed(n)
    t = torch.randn(n, n, dtype=torch.float64, device=dev, generator=g) / n
    t.diagonal().add_(1.0)
    if n == 129:
        t[70, 70] = 2.0 ** -600                  # one block is divided in turn
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    ks = (3 * sms // 2, 3 * sms // 2 + 1, 4 * sms + 3, 8 * sms + 1) if n < 4000 else (3 * sms // 2,)
    b = torch.randn(max(ks), n, dtype=torch.float64, device=dev, generator=g)
    args = dict(lower=lower, trans=trans, unit=unit)
    some = torch.cat([_dense.trsv(t, b[i:i + 40], **args) for i in range(0, max(ks), 40)])
    for k in ks:
        assert torch.equal(_dense.trsv(t, b[:k], **args), some[:k])


def test_getrs_many_vectors_of_several_systems(dev):
    n, bt, k = 180, 5, 61                        # 305 vectors in all, an odd count per system
    g = torch.Generator(device=dev).manual_seed(1)
    a = torch.randn(bt, n, n, dtype=torch.float64, device=dev, generator=g)
    b = torch.randn(bt, k, n, dtype=torch.float64, device=dev, generator=g)
    lu, piv, _ = _dense.lu_factor_batched(a)
    for trans in (0, 1):
        x = _dense.lu_solve_batched(lu, piv, b, trans)
        for s in range(bt):
            assert torch.equal(x[s], _dense.lu_solve_batched(lu[s:s + 1], piv[s:s + 1], b[s:s + 1],
                                                             trans)[0])


@pytest.mark.parametrize("n", [169, 192, 193, 257, 600])
@pytest.mark.parametrize("k", [1, 2, 3, 9, 63, 64])
def test_trsm_many_systems_same_bits_as_each_alone(dev, n, k):
    """Batches of systems with few vectors each, up to and past the count from which they
    are taken to share their matrix, and past eight vectors per SM; one diagonal block
    that is divided in turn."""
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    bt = -(-max(9 * sms, 4 * k) // k) if n < 600 else -(-2 * sms // k)
    g = torch.Generator(device=dev).manual_seed(n + k)
    t = torch.randn(bt, n, n, dtype=torch.float64, device=dev, generator=g) / n
    t.diagonal(dim1=-2, dim2=-1).add_(1.0)
    t[1, 40, 40] = 2.0 ** -600
    piv = torch.arange(n, dtype=torch.int32, device=dev).expand(bt, n).contiguous()
    b = torch.randn(bt, k, n, dtype=torch.float64, device=dev, generator=g)
    for trans in (0, 1):
        x = _dense.lu_solve_batched(t, piv, b, trans)
        for s in (0, 1, 2, bt - 1):
            assert torch.equal(x[s], _dense.lu_solve_batched(t[s:s + 1], piv[s:s + 1],
                                                             b[s:s + 1], trans)[0])


@pytest.mark.parametrize("trans", [0, 1])
def test_getrs_one_vector_per_system_costs_less_than_two(dev, trans):
    """1300 systems of 300 unknowns: with one right-hand side each no more than 0.85 of the
    time with two (as pairs with one half empty it was the same)."""
    n, bt = 300, 1300
    g = torch.Generator(device=dev).manual_seed(2)
    t = torch.randn(bt, n, n, dtype=torch.float64, device=dev, generator=g) / n
    t.diagonal(dim1=-2, dim2=-1).add_(1.0)
    piv = torch.arange(n, dtype=torch.int32, device=dev).expand(bt, n).contiguous()
    best = {}
    for k in (1, 2):
        b = torch.ones(bt, k, n, dtype=torch.float64, device=dev)
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            _dense.lu_solve_batched(t, piv, b, trans)
            e[1].record()
            torch.cuda.synchronize()
            best[k] = min(best.get(k, 1e9), e[0].elapsed_time(e[1]))
    assert best[1] <= 0.85 * best[2]


@pytest.mark.parametrize("n", [2, 3, 8, 31, 32])
@pytest.mark.parametrize("lower", [True, False])
def test_trsm_one_block_rounds_each_unknown(dev, n, lower):
    """Up to 32 unknowns: substitution with each unknown rounded once before it is used,
    x_t = v_t / t_tt and v_l = fma(-t_lt, x_t, v_l), bit for bit (the FMA in extended
    precision: a product of two 53-bit values and one sum, rounded once)."""
    if np.finfo(np.longdouble).nmant < 106:
        pytest.skip("needs quadruple precision on the host for the exact FMA")
    rng = np.random.default_rng(n)
    m = rng.standard_normal((n, n))
    m[np.arange(n), np.arange(n)] += np.sign(m[np.arange(n), np.arange(n)])
    b = rng.standard_normal((40, n))
    order = np.arange(n) if lower else np.arange(n)[::-1]
    for nv in (1, 40):
        x = _dense.trsv(_t(m, dev), _t(b[:nv], dev), lower=lower, trans=False, unit=False)
        v = b[:nv].copy()
        for i, t in enumerate(order):
            v[:, t] = v[:, t] / m[t, t]
            for r in order[i + 1:]:
                v[:, r] = (v[:, r].astype(np.longdouble) -
                           np.longdouble(m[r, t]) * v[:, t].astype(np.longdouble)).astype(np.float64)
        np.testing.assert_array_equal(x.cpu().numpy(), v)
