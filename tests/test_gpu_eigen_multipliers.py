"""Inverse iteration of the large sectors keeps every bit of the elimination's multipliers.

``tt_sym_eigvecs_batched`` on T = tridiag(e, -2e, e), which is its own tridiagonal form
(no reflectors), with the "eigenvalue" 0: the vector that comes out is then T^-3 applied
to the solver's start vector, normalised, and T^-1 is known in closed form (evaluated in
80 bits).  The rounding of the multipliers e / pivot, which approach -1, is what its
error consists of.  The elimination carried out step by step in FP64 on these inputs ends
3.6e-12 and 1.0e-12 away (4096 rows, e = -1 and -0.9), relative to the entries' mean
square; with multipliers of 52 bits 8.9e-11 and 1.0e-10.  The tolerance lies between: 2e-11.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


def _start(n):
    """The solver's start for vector 0 of the first problem: splitmix64 of the row, in [-1, 1)."""
    z = np.arange(n, dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    return (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53 * 2.0 - 1.0


def _exact(n):
    x, i = _start(n).astype(np.longdouble), np.arange(1, n + 1, dtype=np.longdouble)
    for _ in range(3):
        left = np.cumsum(i * x)
        right = np.concatenate([np.cumsum(((n + 1 - i) * x)[::-1])[::-1][1:], [np.longdouble(0)]])
        x = ((n + 1 - i) * left + i * right) / (n + 1)
        x /= np.sqrt(np.sum(x * x))
    return x


@pytest.mark.parametrize("n,e,tol", [(4096, -1.0, 2e-11), (4096, -0.9, 2e-11)])
def test_vector_of_a_chain(n, e, tol):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvecs_batched.restype = C.c_int
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    ctx = tt_b200.Context(0)
    try:
        T = torch.tensor(np.concatenate([np.full(n, -2.0 * e), np.full(n - 1, e), np.zeros(n + 1)]), device="cuda")
        G, Z, w = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (n * n, n * n, n))
        work = torch.zeros(3 * n * n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvecs_batched(ctx.h, (EigProblem * 1)(EigProblem(0, 0, 0, n, 0)), 1, (C.c_int * 1)(1),
                                          G.data_ptr(), T.data_ptr(), w.data_ptr(), Z.data_ptr(), work.data_ptr(),
                                          None) == 0
        ctx.sync()
        got = Z[:n].cpu().numpy()
    finally:
        ctx.close()
    want = _exact(n)
    got = got * np.sign(float(got @ want.astype(np.float64)))
    assert float(np.abs(got - want).max() * np.sqrt(n)) <= tol
