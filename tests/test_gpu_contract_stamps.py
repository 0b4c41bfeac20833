"""The device clock that FP64 contractions and Davidson steps write (tt_contract_exec_stamped,
tt_plan_stamps, tt_dav_stamp_slots, tt_dav_read_stamped).

A launch's stamp is the time at which the work before it has ended, so the difference of two
launches' stamps is the first one's duration.  Contractions of about a millisecond, so that
the clock's resolution (1 us here) and the launches do not matter: within 10 % of what events
around the same contraction say, whichever kernel it runs on.  Only FP64 plans that launch
something take a stamp.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P, I = C.c_void_p, C.c_int
MAXM = 6
OUT = np.dtype([("c_off", "i8"), ("m", "i4"), ("n", "i4"), ("ldc", "i4")], align=True)
PAIR = np.dtype([("out_block", "i4"), ("n_m", "i4"), ("n_k", "i4"), ("n_n", "i4"), ("a_off", "i8"), ("b_off", "i8"),
                 ("m_dims", "i4", MAXM), ("k_dims", "i4", MAXM), ("n_dims", "i4", MAXM), ("a_m_stride", "i8", MAXM),
                 ("a_k_stride", "i8", MAXM), ("b_k_stride", "i8", MAXM), ("b_n_stride", "i8", MAXM)], align=True)


def _lib():
    import tt_b200
    lib = tt_b200.lib
    lib.tt_contract_plan.argtypes = [P, P, I, P, I, I, C.POINTER(P)]
    lib.tt_contract_exec_stamped.argtypes = [P] * 5 + [C.c_double, I, P]
    lib.tt_contract_exec.argtypes = [P] * 5 + [C.c_double]
    lib.tt_plan_stamps.argtypes = [P]
    lib.tt_plan_destroy.argtypes = [P] * 2
    lib.tt_event_create.argtypes = [P, C.POINTER(P)]
    lib.tt_event_record.argtypes = [P, P]
    lib.tt_event_elapsed_ms.argtypes = [P, P, C.POINTER(C.c_float)]
    lib.tt_event_destroy.argtypes = [P]
    lib.tt_dav_state_create.argtypes = [P, C.POINTER(P)]
    lib.tt_dav_state_destroy.argtypes = [P, P]
    lib.tt_dav_stamp_slots.argtypes = [P, I, C.POINTER(P)]
    lib.tt_dav_read_stamped.argtypes = [P, P, P, P]
    lib.tt_dav_step.argtypes = [P, P, I, I, C.c_double, I, C.c_int64, C.POINTER(P), C.POINTER(P), P, P, I, P, C.c_uint64]
    return tt_b200, lib


def _plan(lib, ctx, m, n, ks, prec=0):
    pad = lambda v: tuple(v) + (0,) * (MAXM - len(v))  # noqa: E731
    pairs, a, b = [], 0, 0
    for k in ks:
        pairs.append((0, 1, 1, 1, a, b, pad([m]), pad([k]), pad([n]), pad([1]), pad([m]), pad([1]), pad([k])))
        a, b = a + m * k, b + k * n
    outs, pairs, h = np.array([(0, m, n, m)], dtype=OUT), np.array(pairs, dtype=PAIR), P()
    assert lib.tt_contract_plan(ctx.h, outs.ctypes.data, 1, pairs.ctypes.data, len(pairs), prec, C.byref(h)) == 0
    return h, a, b


@pytest.mark.parametrize("m,n,ks", [(3000, 3000, [1500]), (1000000, 4, [64] * 8), (1000000, 30, [64] * 4),
                                    (700, 500, [60000])])
def test_stamps_against_events(m, n, ks):
    import torch
    tt_b200, lib = _lib()
    ctx = tt_b200.Context(0)
    try:
        h, a, b = _plan(lib, ctx, m, n, ks)
        assert lib.tt_plan_stamps(h) == 1
        A, B = (torch.randn(s, dtype=torch.float64, device="cuda") for s in (a, b))
        out, t = torch.empty(m * n, dtype=torch.float64, device="cuda"), torch.zeros(8, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ev = [P(), P()]
        for e in ev:
            assert lib.tt_event_create(ctx.h, C.byref(e)) == 0
        run = lambda slot: lib.tt_contract_exec_stamped(ctx.h, h, A.data_ptr(), B.data_ptr(),  # noqa: E731
                                                        out.data_ptr(), 1.0, 0, slot)
        for i in range(8):
            assert run(t.data_ptr() + 8 * i) == 0
        ctx.sync()
        ms = []
        for _ in range(5):
            assert lib.tt_event_record(ctx.h, ev[0]) == 0 and run(None) == 0 and lib.tt_event_record(ctx.h, ev[1]) == 0
            ctx.sync()
            x = C.c_float()
            assert lib.tt_event_elapsed_ms(ev[0], ev[1], C.byref(x)) == 0
            ms.append(x.value)
        for e in ev:
            lib.tt_event_destroy(e)
        lib.tt_plan_destroy(ctx.h, h)
    finally:
        ctx.close()
    d = np.diff(t.cpu().numpy().astype(np.float64))[1:] * 1e-6
    assert np.all(d > 0) and abs(np.median(d) / np.median(ms) - 1.0) <= 0.1, (d, ms)


def test_plans_without_a_stamp():
    tt_b200, lib = _lib()
    ctx = tt_b200.Context(0)
    try:
        import torch
        x = torch.zeros(128 * 128, dtype=torch.float64, device="cuda")
        t = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for args, prec in (((128, 128, [128]), 2), ((0, 5, [3]), 0)):
            h, _, _ = _plan(lib, ctx, *args, prec)
            assert lib.tt_plan_stamps(h) == 0
            assert lib.tt_contract_exec_stamped(ctx.h, h, x.data_ptr(), x.data_ptr(), x.data_ptr(), 1.0, 0,
                                                t.data_ptr()) != 0
            lib.tt_plan_destroy(ctx.h, h)
        ctx.sync()
        assert int(t[0]) == 0
    finally:
        ctx.close()


def test_stamps_of_a_loop():
    """Slots 0..2 of a product by its contractions, slot 3 by the step behind it, in order."""
    import torch
    tt_b200, lib = _lib()
    ctx = tt_b200.Context(0)
    try:
        n = 1000
        h, _, _ = _plan(lib, ctx, n, 1, [n])
        A = torch.randn(n, n, dtype=torch.float64, device="cuda")
        A = ((A + A.T) / 100).contiguous()
        v = [torch.randn(n, dtype=torch.float64, device="cuda")]
        v[0] /= v[0].norm()
        tmp, x, va = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"), []
        ranges, st = torch.tensor([0, n], device="cuda"), P()
        torch.cuda.synchronize()
        assert lib.tt_dav_state_create(ctx.h, C.byref(st)) == 0
        ptrs = lambda ts: (P * len(ts))(*[q.data_ptr() for q in ts])  # noqa: E731
        for i in range(3):
            slots = P()
            assert lib.tt_dav_stamp_slots(st, i, C.byref(slots)) == 0
            va.append(torch.zeros_like(x))
            v.append(torch.zeros_like(x))
            torch.cuda.synchronize()
            for k, y in enumerate((tmp, tmp, va[i])):
                assert lib.tt_contract_exec_stamped(ctx.h, h, A.data_ptr(), v[i].data_ptr(), y.data_ptr(), 1.0, 0,
                                                    slots.value + 8 * k) == 0
            assert lib.tt_dav_step(ctx.h, st, i, 2, 1e-30, n, n, ptrs(v[:i + 1]), ptrs(va), x.data_ptr(),
                                   v[i + 1].data_ptr(), 1, ranges.data_ptr(), i) == 0
        res, t = (C.c_double * 8)(), np.zeros((16, 4), dtype=np.uint64)
        assert lib.tt_dav_read_stamped(ctx.h, st, res, t.ctypes.data) == 0
        lib.tt_dav_state_destroy(ctx.h, st)
        lib.tt_plan_destroy(ctx.h, h)
    finally:
        ctx.close()
    t = t[:3].reshape(-1).astype(np.int64)
    assert t[0] > 0 and np.all(np.diff(t) >= 0) and t[-1] > t[0], t
