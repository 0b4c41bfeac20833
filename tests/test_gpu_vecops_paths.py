"""The Davidson vector kernels at every number of vectors and at odd lengths.

Each kernel has one instance per number of vectors up to 8 and one for more, walks pairs
of elements several at a time and leaves an odd last element to one thread
(qtensor/qtensor.cpp:1031-1179).  Overlaps and norms against numpy in extended precision
(sums of n <= 3e5 products of numbers below 1: 1e-12 relative to the sum of their
magnitudes); the projection and the Ritz vector with its residual bit for bit against the
linear combinations whose order of sums they promise, on and off 16-byte boundaries.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lib():
    import tt_b200
    lib, P, I, I64, D = tt_b200.lib, C.c_void_p, C.c_int, C.c_int64, C.c_double
    lib.tt_vec_multidot.argtypes = [P, I64, I, C.POINTER(P), P, P]
    lib.tt_vec_nrm2.argtypes = [P, I64, P, P]
    lib.tt_vec_lincomb_dev.argtypes = [P, I64, I, C.POINTER(P), P, D, I, P]
    lib.tt_vec_project_nrm2_dev.argtypes = [P, I64, I, C.POINTER(P), P, P, P]
    lib.tt_vec_ritz_residual_dev.argtypes = [P, I64, I, C.POINTER(P), C.POINTER(P), P, P, P, P]
    return tt_b200, lib


def _ptrs(ts):
    return (C.c_void_p * max(1, len(ts)))(*[t.data_ptr() for t in ts])


@pytest.mark.parametrize("n", [1, 2, 3, 513, 1024, 4099, 303105, 1212417])
def test_vector_counts(n):
    import torch
    tt_b200, lib = _lib()
    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda k: torch.rand(k, dtype=torch.float64, device="cuda", generator=g) - 0.5  # noqa: E731
    vs, ws = [rand(n) for _ in range(16)], [rand(n) for _ in range(16)]
    off = [rand(n + 1)[1:] for _ in range(2)]  # 8 bytes past a 16-byte boundary
    y0, coef, cq = rand(n), rand(16), rand(17)
    hv, hy = np.stack([v.cpu().numpy() for v in vs]).astype(np.longdouble), y0.cpu().numpy().astype(np.longdouble)
    ctx = tt_b200.Context(0)
    try:
        for nv in range(1, 17):
            out, nrm, nrm2 = (torch.zeros(16, dtype=torch.float64, device="cuda") for _ in range(3))
            y, z = y0.clone(), y0.clone()
            x1, q1, x2, q2, x3, q3 = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(6))
            torch.cuda.synchronize()
            assert lib.tt_vec_multidot(ctx.h, n, nv, _ptrs(vs), y0.data_ptr(), out.data_ptr()) == 0
            assert lib.tt_vec_project_nrm2_dev(ctx.h, n, nv, _ptrs(vs), coef.data_ptr(), y.data_ptr(),
                                               nrm.data_ptr()) == 0
            assert lib.tt_vec_lincomb_dev(ctx.h, n, nv, _ptrs(vs), coef.data_ptr(), -1.0, 1, z.data_ptr()) == 0
            assert lib.tt_vec_nrm2(ctx.h, n, z.data_ptr(), nrm2.data_ptr()) == 0
            if nv < 16:
                assert lib.tt_vec_ritz_residual_dev(ctx.h, n, nv, _ptrs(vs), _ptrs(ws), coef.data_ptr(),
                                                    cq.data_ptr(), x1.data_ptr(), q1.data_ptr()) == 0
                # off the boundary: the last vector is elsewhere
                off[0].copy_(vs[nv - 1])
                off[1].copy_(ws[nv - 1])
                torch.cuda.synchronize()
                assert lib.tt_vec_ritz_residual_dev(ctx.h, n, nv, _ptrs(vs[:nv - 1] + off[:1]),
                                                    _ptrs(ws[:nv - 1] + off[1:]), coef.data_ptr(), cq.data_ptr(),
                                                    x2.data_ptr(), q2.data_ptr()) == 0
                assert lib.tt_vec_lincomb_dev(ctx.h, n, nv, _ptrs(vs), coef.data_ptr(), 1.0, 0, x3.data_ptr()) == 0
                assert lib.tt_vec_lincomb_dev(ctx.h, n, nv + 1, _ptrs(ws[:nv] + [x3]), cq.data_ptr(), 1.0, 0,
                                              q3.data_ptr()) == 0
            ctx.sync()
            ref = hv[:nv] @ hy
            mag = np.abs(hv[:nv]) @ np.abs(hy)
            assert np.all(np.abs(out[:nv].cpu().numpy() - ref) <= 1e-12 * mag), nv
            assert torch.equal(y, z) and torch.equal(nrm[:1], nrm2[:1]), nv
            for a, b, c in ((x1, x2, x3), (q1, q2, q3)):
                assert torch.equal(a, b) and torch.equal(a, c), nv
    finally:
        ctx.close()
