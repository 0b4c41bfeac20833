"""Orthonormality of the eigenvectors of cluster-sized sectors whose inverse-iteration
vectors are far from orthogonal.

A zero density matrix (every eigenvalue equal) leaves the random start vectors as they
are, so all of the orthonormality comes from CholeskyQR2: condition numbers of about
1e3, hence about 1e-11 after its first pass and rounding (a few 1e-15, bound 1e-13)
after its second.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


@pytest.mark.parametrize("n", [161, 200, 333])
def test_equal_eigenvalues(n):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    ctx = tt_b200.Context(0)
    try:
        z = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")  # noqa: E731
        G, Z, T, w, work = z(n * n), z(n * n), z(3 * n), z(n), z(3 * n * n)
        torch.cuda.synchronize()
        prob = (EigProblem * 1)(EigProblem(0, 0, 0, n, 0))
        assert lib.tt_sym_eigvals_batched(ctx.h, prob, 1, G.data_ptr(), T.data_ptr(), w.data_ptr(), None) == 0
        assert lib.tt_sym_eigvecs_batched(ctx.h, prob, 1, (C.c_int * 1)(n), G.data_ptr(), T.data_ptr(), w.data_ptr(),
                                          Z.data_ptr(), work.data_ptr(), None) == 0
        ctx.sync()
        V = Z.cpu().numpy().reshape(n, n)
    finally:
        ctx.close()
    assert np.all(w.cpu().numpy() == 0.0)
    assert np.abs(V @ V.T - np.eye(n)).max() <= 1e-13
