"""The dense Davidson where there is no further direction.

linalg/tensor_davidson.cpp:74-184 normalises every preconditioned residual.  Inside a
restart the residual can vanish (the start is an eigenvector up to a component that one
step removes) and the basis can come to span the space (fewer elements than steps); the
restart then ends with the Ritz vector that it has, the later steps are no-ops, and the
result is an eigenpair to rounding (1e-11, as for the other steps of this loop).
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-11


def _restart(A, D, start, m, high=0):
    """One restart of m steps on the symmetric matrix A; returns the Ritz value, the residual's norm, x and v[0]."""
    import torch
    import tt_b200
    lib, P, I = tt_b200.lib, C.c_void_p, C.c_int
    lib.tt_dav_state_create.argtypes = [P, C.POINTER(P)]
    lib.tt_dav_state_destroy.argtypes = [P, P]
    lib.tt_dav_step_dense.argtypes = [P, P, I, I, I, C.c_int64, C.POINTER(P), C.POINTER(P), P, P]
    lib.tt_dav_read_dense.argtypes = [P, P, C.POINTER(C.c_double), C.POINTER(C.c_double)]
    ptrs = lambda ts: (P * len(ts))(*[t.data_ptr() for t in ts])  # noqa: E731
    A, D, start = (torch.tensor(np.asarray(t, dtype=np.float64), device="cuda") for t in (A, D, start))
    ctx = tt_b200.Context(0)
    try:
        st = P()
        assert lib.tt_dav_state_create(ctx.h, C.byref(st)) == 0
        v = [start / start.norm()] + [torch.full_like(start, float("nan")) for _ in range(m - 1)]
        va, x = [], torch.full_like(start, float("nan"))
        for j in range(m):
            va.append(A @ v[j])
            torch.cuda.synchronize()
            assert lib.tt_dav_step_dense(ctx.h, st, j, m, high, len(start), ptrs(v), ptrs(va), D.data_ptr(),
                                         x.data_ptr()) == 0
            ctx.sync()
        ev, rn = C.c_double(), C.c_double()
        assert lib.tt_dav_read_dense(ctx.h, st, C.byref(ev), C.byref(rn)) == 0
        lib.tt_dav_state_destroy(ctx.h, st)
    finally:
        ctx.close()
    return ev.value, rn.value, x.cpu().numpy(), v[0].cpu().numpy()


def _check(A, ev, rn, x, v0):
    assert np.all(np.isfinite(x)) and np.isfinite(ev) and np.isfinite(rn), (ev, rn, x)
    assert abs(np.linalg.norm(x) - 1.0) <= TOL and np.abs(v0 - x / np.linalg.norm(x)).max() <= TOL
    assert np.abs(A @ x - ev * x).max() <= TOL and rn <= TOL


@pytest.mark.parametrize("m", [1, 2, 3, 6])
@pytest.mark.parametrize("start", [(1.0, 0.0, 1e-16, 0.0), (0.0, 1.0, 0.0, 0.0), (0.6, 0.8, 0.0, 0.0)])
def test_start_is_an_eigenvector(start, m):
    A = np.diag([-1.0, -1.0, 1.0, 1.0])
    ev, rn, x, v0 = _restart(A, np.diag(A), start, m)
    _check(A, ev, rn, x, v0)
    assert abs(ev + 1.0) <= TOL


@pytest.mark.parametrize("high", [0, 1])
@pytest.mark.parametrize("n,m", [(1, 1), (1, 3), (2, 3), (3, 9), (7, 16), (15, 16)])
def test_more_steps_than_elements(n, m, high):
    rng = np.random.default_rng(10 * n + m)
    A = rng.standard_normal((n, n))
    A = A + A.T
    A /= np.linalg.norm(A, 2)
    ev, rn, x, v0 = _restart(A, np.zeros(n), rng.standard_normal(n), m, high)
    _check(A, ev, rn, x, v0)
    assert abs(ev - np.linalg.eigvalsh(A)[-1 if high else 0]) <= TOL


@pytest.mark.parametrize("L,maxm,sweeps", [(6, 16, 3), (20, 512, 2)])
def test_sweeps_from_an_eigenstate(L, maxm, sweeps):
    """The Ising chain from its ground state; with every singular value kept, 20 sites reach vectors of 512 x 4 x 512
    elements, which the host's loop handles."""
    import tt_b200
    a = tt_b200.AutoMPO()
    for i in range(L - 1):
        a.add(-1.0, "Sz", i, "Sz", i + 1)
    ctx = tt_b200.Context(0)
    try:
        psi = tt_b200.DMPS(L, [1] * L)
        H = tt_b200.DMPO.from_autompo(a, L)
        e, se, _ = tt_b200.ddmrg_run(psi, H, sweeps, [maxm], [0.0], [2])
        del psi, H
    finally:
        ctx.close()
    assert np.all(np.abs(np.array(se + [e]) + 0.25 * (L - 1)) <= 1e-10), (se, e)
