"""Eigenvectors of cluster-sized sectors at the remainders of their kernels' tiles.

CholeskyQR2 and the back-transformation work on panels of 32 vectors, 32 rows and 32
reflectors, on vectors 16 at a time and rows 8 at a time: one vector, one less and one
more than a panel, every vector of a sector, several sectors with different numbers in
one call (svd_bond keeps the largest states of all sectors, qtensor/qtensor_op.cpp
:1229-1300).  Density-matrix-like and rank-deficient spectra; the tolerances of the other
eigensolver tests: residuals and orthonormality 1e-10.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


@pytest.mark.parametrize("kind", ["decay", "rank"])
@pytest.mark.parametrize("ns,nvec", [([129, 129, 130, 131], [1, 31, 0, 131]), ([136, 137, 160], [32, 33, 160]),
                                     ([258, 259], [65, 259]), ([513], [479]), ([769, 140], [769, 17])])
def test_remainders(ns, nvec, kind):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.restype = lib.tt_sym_eigvecs_batched.restype = C.c_int
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    rng = np.random.default_rng(sum(ns))
    mats = []
    for n in ns:
        Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        lam = np.exp(-np.linspace(0.0, 32.0, n)) * rng.uniform(0.5, 1.0, n)
        if kind == "rank":
            lam[n // 3:] = 0.0
        M = (Q * lam) @ Q.T
        mats.append(0.5 * (M + M.T))
    g_off = np.concatenate([[0], np.cumsum([n * n for n in ns])]).astype(np.int64)
    w_off = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    probs = (EigProblem * len(ns))(*[EigProblem(int(g), int(w), 0, n, 0) for g, w, n in zip(g_off, w_off, ns)])
    ctx = tt_b200.Context(0)
    try:
        G = torch.tensor(np.concatenate([m.reshape(-1) for m in mats]), device="cuda")
        T, w = (torch.zeros(k * int(w_off[-1]), dtype=torch.float64, device="cuda") for k in (3, 1))
        Z = torch.full((int(g_off[-1]),), float("nan"), dtype=torch.float64, device="cuda")
        work = torch.full((3 * int(g_off[-1]),), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvals_batched(ctx.h, probs, len(ns), G.data_ptr(), T.data_ptr(), w.data_ptr(), None) == 0
        assert lib.tt_sym_eigvecs_batched(ctx.h, probs, len(ns), (C.c_int * len(ns))(*nvec), G.data_ptr(),
                                          T.data_ptr(), w.data_ptr(), Z.data_ptr(), work.data_ptr(), None) == 0
        ctx.sync()
        wh, Zh = w.cpu().numpy(), Z.cpu().numpy()
    finally:
        ctx.close()
    for p, (M, n, k) in enumerate(zip(mats, ns, nvec)):
        if k == 0:
            continue
        V = Zh[g_off[p]:g_off[p] + n * k].reshape(n, k, order="F")
        assert np.linalg.norm(M @ V - V * wh[w_off[p]:w_off[p] + k], axis=0).max() <= 1e-10, n
        assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-10, n
