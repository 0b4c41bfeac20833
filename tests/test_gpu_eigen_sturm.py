"""Eigenvalue counts of the library on matrices that are already tridiagonal.

``tt_sym_eigvals_batched`` bisects on Sturm counts of T scaled to a norm below 1, with the
off-diagonals floored and the pair of minors rescaled every eight steps (sturm_count in
csrc/tridiag_eig.cu).  T here is what the reduction starts from: split into blocks by zero
off-diagonals, constant over long stretches, with entries that the bisection points hit
exactly, graded, of norm 1e6 and 1e-9, at sizes of the one-CTA and the cluster reduction.
Reference: LAPACK (numpy eigvalsh); 1e-12 ||T|| as in the other eigenvalue tests.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


def _tridiagonals(n, rng):
    k = np.arange(n, dtype=float)
    yield np.full(n, 2.0), np.full(n - 1, -1.0)                              # a Laplacian
    yield np.zeros(n), np.ones(n - 1)                                        # symmetric spectrum, zero diagonal
    d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
    e[rng.integers(0, n - 1, n // 3)] = 0.0
    yield d, e                                                               # split at random places
    yield np.where(k < n // 2, 1.0, 0.25), np.zeros(n - 1)                   # diagonal, two values
    yield np.repeat(rng.standard_normal(n // 8 + 1), 8)[:n], np.tile([0.5] * 7 + [0.0], n // 8 + 1)[:n - 1]
    yield 10.0 ** (-k / n * 12), 10.0 ** (-k[:-1] / n * 12) * 0.3            # graded
    yield np.abs(k - n // 2), np.ones(n - 1)                                 # Wilkinson's, pairs equal to rounding


@pytest.mark.parametrize("scale", [1.0, 1e6, 1e-9])
@pytest.mark.parametrize("n", [2, 9, 33, 128, 129, 500])
def test_spectra(n, scale):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.restype = C.c_int
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    mats = [scale * (np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
            for d, e in _tridiagonals(n, np.random.default_rng(n))]
    probs = (EigProblem * len(mats))(*[EigProblem(i * n * n, i * n, 0, n, 0) for i in range(len(mats))])
    ctx = tt_b200.Context(0)
    try:
        G = torch.tensor(np.concatenate([m.reshape(-1) for m in mats]), device="cuda")
        T, w = (torch.zeros(k * n * len(mats), dtype=torch.float64, device="cuda") for k in (3, 1))
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvals_batched(ctx.h, probs, len(mats), G.data_ptr(), T.data_ptr(), w.data_ptr(), None) == 0
        ctx.sync()
        got = w.cpu().numpy().reshape(len(mats), n)
    finally:
        ctx.close()
    for i, M in enumerate(mats):
        assert np.abs(got[i] - np.linalg.eigvalsh(M)[::-1]).max() <= 1e-12 * np.linalg.norm(M, 2), i
