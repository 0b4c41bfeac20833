"""The narrow FP64 contractions (output blocks of at most 32 columns, short k per pair) on
the routes that single small blocks do not take.

Through ``tt_contract_plan`` / ``tt_contract_exec`` (the inner loop of qtensor::operator*,
qtensor/qtensor.cpp:652-726) against FP64 matrix products by torch; an element that sums K
products may differ by the rounding of two summation orders, at most 2 K 2^-53 sum |a b|.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAXM = 6
OUT = np.dtype([("c_off", "i8"), ("m", "i4"), ("n", "i4"), ("ldc", "i4")], align=True)
PAIR = np.dtype([("out_block", "i4"), ("n_m", "i4"), ("n_k", "i4"), ("n_n", "i4"), ("a_off", "i8"), ("b_off", "i8"),
                 ("m_dims", "i4", MAXM), ("k_dims", "i4", MAXM), ("n_dims", "i4", MAXM), ("a_m_stride", "i8", MAXM),
                 ("a_k_stride", "i8", MAXM), ("b_k_stride", "i8", MAXM), ("b_n_stride", "i8", MAXM)], align=True)


@pytest.fixture(scope="module")
def ctx():
    import tt_b200
    c = tt_b200.Context(0)
    yield c
    c.close()


def _pad(v):
    return tuple(v) + (0,) * (MAXM - len(v))


def _exec(ctx, outs, pairs, A, B, c_size, alpha=1.0):
    import torch
    import tt_b200
    lib, P = tt_b200.lib, C.c_void_p
    lib.tt_contract_plan.restype = lib.tt_contract_exec.restype = C.c_int
    lib.tt_contract_plan.argtypes = [P, P, C.c_int, P, C.c_int, C.c_int, C.POINTER(P)]
    lib.tt_contract_exec.argtypes = [P] * 5 + [C.c_double]
    lib.tt_plan_destroy.argtypes = [P] * 2
    outs, pairs, h = np.array(outs, dtype=OUT), np.array(pairs, dtype=PAIR), P()
    out = torch.full((c_size,), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.tt_contract_plan(ctx.h, outs.ctypes.data, len(outs), pairs.ctypes.data, len(pairs), 0,
                                C.byref(h)) == 0, lib.tt_get_last_error()
    try:
        for _ in range(2):
            assert lib.tt_contract_exec(ctx.h, h, A.data_ptr(), B.data_ptr(), out.data_ptr(), alpha) == 0
        ctx.sync()
    finally:
        lib.tt_plan_destroy(ctx.h, h)
    return out


def test_offsets_beyond_31_bits(ctx):
    """A block of B whose rows and columns reach 2^31 elements only together."""
    import torch
    m, ks, cs = 300, 2 ** 31 - 64, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(2 * m, dtype=torch.float64, device="cuda", generator=g)
    B = torch.empty(ks + cs + 1, dtype=torch.float64, device="cuda")
    b = torch.randn(2, 2, dtype=torch.float64, device="cuda", generator=g)
    for k in range(2):
        for c in range(2):
            B[k * ks + c * cs] = b[k, c]
    out = _exec(ctx, [(0, m, 2, m)], [(0, 1, 1, 1, 0, 0, _pad([m]), _pad([2]), _pad([2]), _pad([1]), _pad([m]),
                                       _pad([ks]), _pad([cs]))], A, B, 2 * m)
    a = A.reshape(2, m).T
    bound = 2 * 2 * 2.0 ** -53 * (a.abs() @ b.abs())
    assert torch.all((out.reshape(2, m).T - a @ b).abs() <= bound)


@pytest.mark.parametrize("kind", ["rows", "rows inner", "columns", "k"])
def test_negative_strides(ctx, kind):
    """Modes walked backwards: the second or the first row mode, B's columns, both operands' k."""
    import torch
    md, k, n = (40, 9), 5, 6
    g = torch.Generator(device="cuda").manual_seed(2)
    A, B = (torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in (3 * 360 * k, 3 * k * n))
    am, ak, bk, bn = [1, 40], [360], [1], [k]
    ao = bo = 0
    if kind == "rows":
        am, ao = [1, -40], 320
    elif kind == "rows inner":
        am, ao = [-1, 40], 39
    elif kind == "columns":
        bn, bo = [-k], k * (n - 1)
    else:
        ak, ao, bk, bo = [-360], 360 * (k - 1), [-1], k - 1
    a = A[:360 * k].reshape(k, 9, 40)
    b = B[:k * n].reshape(n, k)
    if kind == "rows":
        a = a.flip(1)
    elif kind == "rows inner":
        a = a.flip(2)
    elif kind == "columns":
        b = b.flip(0)
    a, b = a.reshape(k, 360).T, b.T
    out = _exec(ctx, [(0, 360, n, 360)], [(0, 2, 1, 1, ao, bo, _pad(md), _pad([k]), _pad([n]), _pad(am), _pad(ak),
                                           _pad(bk), _pad(bn))], A, B, 360 * n, alpha=-0.5)
    bound = 2 * k * 2.0 ** -53 * 0.5 * (a.abs() @ b.abs())
    assert torch.all((out.reshape(n, 360).T + 0.5 * (a @ b)).abs() <= bound)
