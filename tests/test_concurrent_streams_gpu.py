"""GPU: factorisations and solves on several streams at once, from as many threads,
against the same calls alone: the same bits.  CTAs of one launch then start at different
times and kernels launched beside one another share the SMs with other work."""

import random
import threading

import pytest
import torch

from lineax_gb300 import _dense, _krylov, mixed
import lineax_gb300 as lx

pytestmark = pytest.mark.gpu


def _calls(dev):
    g = torch.Generator(device=dev).manual_seed(7)

    def rand(*shape):
        return torch.randn(*shape, dtype=torch.float64, device=dev, generator=g)

    def spd(n):
        x = rand(n, n)
        return x @ x.T / n + torch.eye(n, dtype=torch.float64, device=dev)

    def lu(a, b):
        f = _dense.lu_factor(a)
        return [*f, _dense.lu_solve(*f, b), _dense.lu_solve(*f, b, 1)]

    def chol(a, b):
        u = _dense.cho_factor(a)
        return [u, _dense.cho_solve(u, b)]

    def qr(a, c):
        f = _dense.geqrf(a)
        return [*f, _dense.ormqr(*f, c, trans=True)]

    def lu32(a, x):
        f = mixed.lu_factor_tf32(a, "3xtf32")
        inv = mixed.lu_inverse(f, "3xtf32")
        return [f.lu, f.piv, inv.linv, inv.uinv, inv.perm,
                mixed.InverseLUPreconditioner(f, inv).mv_block(x)]

    def chol32(a):
        f = mixed.cholesky_factor_tf32(a)
        return [f.lu, mixed.cholesky_inverse(f).linv]

    def qr32(a):
        q = mixed.qr_square_tf32(a)
        return [q.qt, q.rinv]

    def gmres(a, b):
        return [_krylov.gmres_run(lx.MatrixLinearOperator(a), b, rtol=1e-9, atol=1e-9).y]

    def cg(b):
        return [_krylov.cg_poisson_mixed(lx.Poisson2DOperator(257, 300), b, rtol=1e-10, atol=1e-10,
                                         max_steps=40).y]

    near = rand(600, 600) * (0.5 / 600 ** 0.5) + torch.eye(600, dtype=torch.float64, device=dev)
    return [(lu, (rand(n, n), rand(k, n))) for n, k in ((168, 5), (517, 3), (1000, 300))] + \
        [(chol, (spd(n), rand(2, n))) for n in (300, 1531)] + \
        [(qr, (rand(m, n), rand(3, m))) for m, n in ((300, 40), (3001, 101))] + \
        [(lu32, (rand(512, 512), rand(9, 512))), (chol32, (spd(1024),)), (qr32, (rand(512, 512),)),
         (gmres, (near, rand(2, 600))), (cg, (rand(4, 257 * 300),))]


def test_calls_on_several_streams_at_once(dev):
    calls = _calls(dev)
    alone = [[t.clone() for t in f(*args)] for f, args in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(seed):
        try:
            rng = random.Random(seed)
            with torch.cuda.device(dev), torch.cuda.stream(torch.cuda.Stream(dev)):
                for i in rng.sample(list(range(len(calls))) * 8, 8 * len(calls)):
                    f, args = calls[i]
                    for j, (x, y) in enumerate(zip(f(*args), alone[i])):
                        if not torch.equal(x, y):
                            wrong.append((f.__name__, tuple(args[0].shape), j))
        except Exception as e:  # reported by the assertion below
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
