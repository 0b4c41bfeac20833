"""Batches of cluster-sized sectors whose number or volume decides how they are reduced.

``tt_sym_eigvals_batched`` / ``tt_sym_eigvecs_batched`` (the per-QN-sector density matrices
of svd_bond, qtensor/qtensor_op.cpp:1229-1300).  Matrices with a known spectrum (a diagonal
between two reflections); tolerances of the other eigensolver tests: eigenvalues 1e-12
||G||, residuals and orthonormality 1e-10.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


def _reflect(G, v):
    g = G @ v
    return G - 2.0 * np.outer(v, g) - 2.0 * np.outer(g, v) + 4.0 * (v @ g) * np.outer(v, v)


@pytest.mark.parametrize("ns", [[1900] * 4 + [130, 40], [2049, 700], [129 + 3 * (i % 11) for i in range(12)],
                                [160, 131, 20] * 9, [129 + i % 32 for i in range(80)], [300] * 18 + [129]])
def test_batch(ns):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.restype = lib.tt_sym_eigvecs_batched.restype = C.c_int
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    rng = np.random.default_rng(len(ns) + ns[0])
    mats, lams = {}, {}
    for n in sorted(set(ns)):  # equal sizes share a matrix
        lams[n] = np.exp(-np.linspace(0.0, 30.0, n))
        G = np.diag(rng.permutation(lams[n]))
        for _ in range(2):
            v = rng.standard_normal(n)
            G = _reflect(G, v / np.linalg.norm(v))
        mats[n] = 0.5 * (G + G.T)
    g_off = np.concatenate([[0], np.cumsum([n * n for n in ns])]).astype(np.int64)
    w_off = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    nvec = [min(n, 40) for n in ns]
    probs = (EigProblem * len(ns))(*[EigProblem(int(g), int(w), 0, n, 0) for g, w, n in zip(g_off, w_off, ns)])
    ctx = tt_b200.Context(0)
    try:
        G = torch.tensor(np.concatenate([mats[n].reshape(-1) for n in ns]), device="cuda")
        T, w = (torch.zeros(k * int(w_off[-1]), dtype=torch.float64, device="cuda") for k in (3, 1))
        Z = torch.full((int(g_off[-1]),), float("nan"), dtype=torch.float64, device="cuda")
        work = torch.zeros(3 * int(g_off[-1]), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.tt_sym_eigvals_batched(ctx.h, probs, len(ns), G.data_ptr(), T.data_ptr(), w.data_ptr(), None) == 0
        assert lib.tt_sym_eigvecs_batched(ctx.h, probs, len(ns), (C.c_int * len(ns))(*nvec), G.data_ptr(),
                                          T.data_ptr(), w.data_ptr(), Z.data_ptr(), work.data_ptr(), None) == 0
        ctx.sync()
        wh, Zh = w.cpu().numpy(), Z.cpu().numpy()
    finally:
        ctx.close()
    for p, (n, k) in enumerate(zip(ns, nvec)):
        got = wh[w_off[p]:w_off[p] + n]
        assert np.abs(got - lams[n]).max() <= 1e-12, (p, n)
        V = Zh[g_off[p]:g_off[p] + n * k].reshape(n, k, order="F")
        assert np.linalg.norm(mats[n] @ V - V * got[:k], axis=0).max() <= 1e-10, (p, n)
        assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-10, (p, n)
