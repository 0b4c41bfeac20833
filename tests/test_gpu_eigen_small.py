"""The block SVD's eigensolver on sectors around the sizes where its kernels change.

``tt_sym_eigvals_batched`` / ``tt_sym_eigvecs_batched`` (the per-QN-sector density
matrices of svd_bond, qtensor/qtensor_op.cpp:1229-1300) on batches of sectors of
1 to 129 states: below and above a row chunk of 32, the largest one-CTA sector
(128) and the smallest cluster-sized one, alone and mixed in one batch, keeping
no, some or all states.  Spectra: density-matrix-like decay, rank-deficient (many
equal zero eigenvalues, whose inverse-iteration vectors collapse onto each other),
exactly degenerate pairs, already diagonal, zero.  Reference: LAPACK (numpy eigh),
with the tolerances of the larger sectors' test: eigenvalues 1e-12 ||G||,
residuals and orthonormality 1e-10.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EigProblem(C.Structure):
    _fields_ = [("g_off", C.c_int64), ("w_off", C.c_int64), ("a_off", C.c_int64),
                ("n", C.c_int32), ("flags", C.c_int32)]


def _matrix(n, rng, kind):
    if kind == "zero":
        return np.zeros((n, n))
    if kind == "diagonal":
        return np.diag(np.exp(-np.linspace(0.0, 20.0, n)))
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    if kind == "decay":
        lam = np.exp(-np.linspace(0.0, np.log(1e14), n)) * rng.uniform(0.5, 1.0, n)
    elif kind == "rank":
        r = max(1, n // 3)
        lam = np.concatenate([np.exp(-np.linspace(0.0, 20.0, r)), np.zeros(n - r)])
    else:
        lam = np.repeat(np.exp(-np.linspace(0.0, 25.0, (n + 1) // 2)), 2)[:n]
    G = (Q * lam) @ Q.T
    return 0.5 * (G + G.T)


def _solve(mats, nvec):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_sym_eigvals_batched.restype = lib.tt_sym_eigvecs_batched.restype = C.c_int
    lib.tt_sym_eigvals_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, P, P, P, P]
    lib.tt_sym_eigvecs_batched.argtypes = [P, C.POINTER(EigProblem), C.c_int, C.POINTER(C.c_int), P, P, P, P, P, P]
    ns = [m.shape[0] for m in mats]
    g_off = np.concatenate([[0], np.cumsum([n * n for n in ns])]).astype(np.int64)
    w_off = np.concatenate([[0], np.cumsum(ns)]).astype(np.int64)
    probs = (EigProblem * len(ns))(*[EigProblem(int(g), int(w), 0, n, 0) for g, w, n in zip(g_off, w_off, ns)])
    ctx = tt_b200.Context(0)
    try:
        G = torch.tensor(np.concatenate([m.reshape(-1, order="F") for m in mats]), device="cuda")
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
    for p, (M, n, k) in enumerate(zip(mats, ns, nvec)):
        gnorm = np.linalg.norm(M, 2)
        got = wh[w_off[p]:w_off[p] + n]
        assert np.all(np.diff(got) <= 0.0)
        assert np.abs(got - np.linalg.eigvalsh(M)[::-1]).max() <= 1e-12 * gnorm, n
        V = Zh[g_off[p]:g_off[p] + n * k].reshape(n, k, order="F")
        if k == 0:
            continue
        assert np.linalg.norm(M @ V - V * got[:k], axis=0).max() <= 1e-10 * gnorm, n
        assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-10, n
        assert np.all(V[np.argmax(np.abs(V), axis=0), np.arange(k)] > 0.0)


SIZES = [1, 2, 3, 5, 31, 32, 33, 64, 65, 96, 127, 128, 129]


@pytest.mark.parametrize("kind", ["decay", "rank", "degenerate", "diagonal", "zero"])
@pytest.mark.parametrize("keep", ["all", "half"])
def test_sizes_in_one_batch(kind, keep):
    rng = np.random.default_rng(11)
    mats = [_matrix(n, rng, kind) for n in SIZES]
    _solve(mats, [n if keep == "all" else n // 2 for n in SIZES])


@pytest.mark.parametrize("n", SIZES)
def test_one_sector(n):
    rng = np.random.default_rng(n)
    _solve([_matrix(n, rng, "decay")], [(2 * n + 2) // 3])


def test_scales_and_mixed_with_large_sectors():
    rng = np.random.default_rng(5)
    mats = [1e-200 * _matrix(40, rng, "decay"), 1e150 * _matrix(17, rng, "rank"), _matrix(300, rng, "decay"),
            _matrix(100, rng, "degenerate")]
    _solve(mats, [20, 17, 120, 100])
