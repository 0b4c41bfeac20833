"""One Davidson iteration in one launch (tt_dav_step, tt_dav_step_dense).

The loops of linalg/tensor_davidson.cpp:74-184 and :193-347 on A = diag(d) + u u^T, the
products by torch, against what the definitions say about the vectors that come out: an
orthonormal basis, the lowest (highest) eigenpair of the projected matrix in it, the
residual's norm, the preconditioned direction.  Lengths around one thread block, the
cluster sizes and the largest that a step takes; 1 to 15 basis vectors; a basis that is
complete, one that a random refill completes.  Sums of n products of unit vectors err by
about sqrt(n) eps <= 1e-13, and the second entries of A reach 3: tolerance 1e-11.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-11


class Result(C.Structure):
    _fields_ = [(k, C.c_int) for k in ("done", "final_ii", "fail_ii", "iters", "randomized")] + [("lam", C.c_double)]


def _lib():
    import tt_b200
    lib, P, I, I64, D = tt_b200.lib, C.c_void_p, C.c_int, C.c_int64, C.c_double
    lib.tt_dav_state_create.argtypes = [P, C.POINTER(P)]
    lib.tt_dav_state_destroy.argtypes = [P, P]
    lib.tt_dav_step.argtypes = [P, P, I, I, D, I, I64, C.POINTER(P), C.POINTER(P), P, P, I, P, C.c_uint64]
    lib.tt_dav_read.argtypes = [P, P, C.POINTER(Result)]
    lib.tt_dav_step_dense.argtypes = [P, P, I, I, I, I64, C.POINTER(P), C.POINTER(P), P, P]
    lib.tt_dav_read_dense.argtypes = [P, P, C.POINTER(D), C.POINTER(D)]
    return tt_b200, lib


class _Problem:
    def __init__(self, n, seed):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.torch, self.n = torch, n
        self.d = torch.linspace(-1.0, 2.0, n, dtype=torch.float64, device="cuda")
        self.u = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
        self.u /= self.u.norm()
        self.start = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
        self.start /= self.start.norm()

    def apply(self, x):
        return self.d * x + self.u * (self.u @ x)


def _ptrs(ts):
    return (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


@pytest.mark.parametrize("n,maxiter", [(2, 1), (3, 2), (33, 4), (511, 13), (512, 3), (1025, 7), (4097, 4),
                                       (16385, 8), (65536, 13), (262143, 3), (262144, 14)])
def test_step(n, maxiter):
    tt_b200, lib = _lib()
    p = _Problem(n, n)
    torch = p.torch
    ctx = tt_b200.Context(0)
    try:
        st = C.c_void_p()
        assert lib.tt_dav_state_create(ctx.h, C.byref(st)) == 0
        v, va = [p.start], [p.apply(p.start)]
        x, ranges = torch.zeros_like(p.start), torch.tensor([0, n], device="cuda")
        for ii in range(maxiter + 1):
            q = torch.full_like(p.start, float("nan"))
            torch.cuda.synchronize()
            assert lib.tt_dav_step(ctx.h, st, ii, maxiter, 1e-30, n, n, _ptrs(v), _ptrs(va), x.data_ptr(),
                                   q.data_ptr(), 1, ranges.data_ptr(), ii) == 0
            ctx.sync()
            if ii < maxiter:
                v.append(q)
                va.append(p.apply(q))
        r = Result()
        assert lib.tt_dav_read(ctx.h, st, C.byref(r)) == 0
        lib.tt_dav_state_destroy(ctx.h, st)
    finally:
        ctx.close()
    V, VA = torch.stack(v).cpu().numpy(), torch.stack(va).cpu().numpy()
    x = x.cpu().numpy()
    assert (r.done, r.final_ii, r.iters, r.randomized) == (1, maxiter, maxiter, 0)
    # one Gram-Schmidt pass each: the residuals here keep at least a few per cent
    assert np.abs(V @ V.T - np.eye(len(V))).max() <= 1e-9
    H = np.tril(V @ VA.T)
    w, Y = np.linalg.eigh(H)
    assert abs(r.lam - w[0]) <= TOL
    y = Y[:, 0] * np.sign(Y[0, 0])
    assert np.abs(x - y @ V).max() <= 1e-9


def test_refill_and_end_of_the_space():
    """The start is an eigenvector: the first residual is rounding, so the new vector is
    drawn at random in the given range and orthogonalised; with maxsize reached the loop ends."""
    tt_b200, lib = _lib()
    torch = _Problem(8, 0).torch
    for maxsize, n in ((700, 700), (1, 700)):
        ctx = tt_b200.Context(0)
        try:
            st = C.c_void_p()
            assert lib.tt_dav_state_create(ctx.h, C.byref(st)) == 0
            v0 = torch.zeros(n, dtype=torch.float64, device="cuda")
            v0[5] = 1.0
            va0 = 0.5 * v0 + 1e-11 * torch.roll(v0, 1)  # residual 1e-11: above the end of the loop, below 1e-10
            x, q = torch.zeros_like(v0), torch.zeros_like(v0)
            ranges = torch.tensor([3, 10, 600, 650], device="cuda")
            torch.cuda.synchronize()
            assert lib.tt_dav_step(ctx.h, st, 0, 3, 1e-30, maxsize, n, _ptrs([v0]), _ptrs([va0]), x.data_ptr(),
                                   q.data_ptr(), 2, ranges.data_ptr(), 7) == 0
            r = Result()
            assert lib.tt_dav_read(ctx.h, st, C.byref(r)) == 0
            lib.tt_dav_state_destroy(ctx.h, st)
        finally:
            ctx.close()
        assert abs(r.lam - 0.5) <= TOL
        if maxsize == 1:
            assert (r.done, r.final_ii, r.fail_ii, r.randomized) == (1, 0, 0, 0)
        else:
            q = q.cpu().numpy()
            assert (r.done, r.randomized) == (0, 1)
            assert abs(np.linalg.norm(q) - 1.0) <= TOL and abs(q[5]) <= TOL
            inside = np.zeros(n, bool)
            inside[3:10] = inside[600:650] = True
            assert np.all(q[~inside] == 0.0) and np.all(q[inside & (np.arange(n) != 5)] > 0.0)


@pytest.mark.parametrize("n,m,high", [(2, 2, 0), (7, 3, 1), (513, 3, 0), (1024, 1, 0), (8193, 5, 1), (16384, 3, 0),
                                      (262144, 9, 0)])
def test_dense_restart(n, m, high):
    tt_b200, lib = _lib()
    p = _Problem(n, n + 1)
    torch = p.torch
    D = p.d + p.u * p.u
    ctx = tt_b200.Context(0)
    try:
        st = C.c_void_p()
        assert lib.tt_dav_state_create(ctx.h, C.byref(st)) == 0
        v = [p.start.clone()] + [torch.full_like(p.start, float("nan")) for _ in range(m - 1)]
        va, x = [], torch.full_like(p.start, float("nan"))
        for j in range(m):
            va.append(p.apply(v[j]))
            torch.cuda.synchronize()
            assert lib.tt_dav_step_dense(ctx.h, st, j, m, high, n, _ptrs(v), _ptrs(va), D.data_ptr(),
                                         x.data_ptr()) == 0
            ctx.sync()
        ev, rn = C.c_double(), C.c_double()
        assert lib.tt_dav_read_dense(ctx.h, st, C.byref(ev), C.byref(rn)) == 0
        lib.tt_dav_state_destroy(ctx.h, st)
    finally:
        ctx.close()
    x, v0 = x.cpu().numpy(), v[0].cpu().numpy()
    V = torch.stack([p.start] + v[1:]).cpu().numpy()  # v[0] now holds the normalised Ritz vector
    VA = torch.stack(va).cpu().numpy()
    assert np.abs(V @ V.T - np.eye(m)).max() <= TOL
    w, Y = np.linalg.eigh(np.tril(V @ VA.T))
    k = m - 1 if high else 0
    assert abs(ev.value - w[k]) <= TOL
    y = Y[:, k] * np.sign((Y[:, k] @ V) @ x)
    assert np.abs(x - y @ V).max() <= 1e-9
    assert np.abs(v0 - x / np.linalg.norm(x)).max() <= TOL
    assert abs(rn.value - np.linalg.norm(y @ VA - w[k] * (y @ V))) <= 1e-9
    if m > 1:  # the first direction: the preconditioned residual, orthogonalised
        th = V[0] @ VA[0]
        t = (VA[0] - th * V[0]) / (D.cpu().numpy() - th)
        t /= np.linalg.norm(t)
        for _ in range(2):
            t -= V[0] * (V[0] @ t)
        assert np.abs(V[1] - t / np.linalg.norm(t)).max() <= 1e-9
