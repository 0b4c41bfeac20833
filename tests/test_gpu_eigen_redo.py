"""Sectors whose eigenvectors the GPU-wide path gives up and the cluster kernel redoes.

``tt_sym_eigvecs_batched`` with one eigenvalue given twice: inverse iteration then gives the
same vector twice and the first Cholesky factorisation of the Gram matrix meets a pivot of
zero.  The flag that it raises in its own launch must not stop part of the cluster that
raises it (shown by reading; every CTA now reads it before one may raise it).  The sector is
redone, the vectors of its other eigenvalues are orthonormal eigenvectors (there is no second
one for the one given twice), and a sector beside it is not redone.  1e-10, as in the other
eigensolver tests.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


@pytest.mark.parametrize("n", [140, 700])
def test_eigenvalue_given_twice(n):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.restype = lib.tt_sym_eigvecs_batched.restype = C.c_int
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    rng, mats, ns = np.random.default_rng(n), [], [n, 150]
    for k in ns:
        Q, _ = np.linalg.qr(rng.standard_normal((k, k)))
        G = (Q * np.linspace(1.0, 2.0, k)) @ Q.T
        mats.append(0.5 * (G + G.T))
    g_off = np.concatenate([[0], np.cumsum([n * n for n in ns])]).astype(np.int64)
    w_off = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    probs = (EigProblem * len(ns))(*[EigProblem(int(g), int(w), 0, n, 0) for g, w, n in zip(g_off, w_off, ns)])
    ctx = tt_b200.Context(0)
    try:
        before = tt_b200.eig_redo_count(ctx)
        G = torch.tensor(np.concatenate([m.reshape(-1) for m in mats]), device="cuda")
        T, w = (torch.zeros(k * int(w_off[-1]), dtype=torch.float64, device="cuda") for k in (3, 1))
        Z = torch.full((int(g_off[-1]),), float("nan"), dtype=torch.float64, device="cuda")
        work = torch.zeros(3 * int(g_off[-1]), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvals_batched(ctx.h, probs, len(ns), G.data_ptr(), T.data_ptr(), w.data_ptr(), None) == 0
        ctx.sync()
        w[n // 2] = w[n // 2 - 1]
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvecs_batched(ctx.h, probs, len(ns), (C.c_int * len(ns))(*ns), G.data_ptr(), T.data_ptr(),
                                          w.data_ptr(), Z.data_ptr(), work.data_ptr(), None) == 0
        ctx.sync()
        wh, Zh = w.cpu().numpy(), Z.cpu().numpy()
        redone = tt_b200.eig_redo_count(ctx) - before
    finally:
        ctx.close()
    assert redone == 1
    for p, (M, k) in enumerate(zip(mats, ns)):
        V, lam = Zh[g_off[p]:g_off[p] + k * k].reshape(k, k, order="F"), wh[w_off[p]:w_off[p] + k]
        if p == 0:
            V, lam = np.delete(V, [n // 2 - 1, n // 2], axis=1), np.delete(lam, [n // 2 - 1, n // 2])
        assert np.linalg.norm(M @ V - V * lam, axis=0).max() <= 1e-10, p
        assert np.abs(V.T @ V - np.eye(len(lam))).max() <= 1e-10, p
