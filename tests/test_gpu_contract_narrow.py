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


def _strides(dims, gap):
    st, run = [], 1
    for d in dims:
        st.append(run)
        run = run * d + gap
    return st, run


def _offsets(dims, st):
    import torch
    r = torch.zeros(1, dtype=torch.int64, device="cuda")
    for d, s in zip(dims, st):
        r = (r[None, :] + (torch.arange(d, device="cuda") * s)[:, None]).reshape(-1)
    return r


def _check(ctx, rows, blocks, alpha=1.0, gap=0, seed=0):
    """blocks: per output block its column modes and the (k modes, key) of its pairs; pairs of one key share their A.
    A holds its row modes (`rows`) first, B its k modes; `gap` unused elements after every mode."""
    import torch
    m, (am, msize) = int(np.prod(rows)), _strides(rows, gap)
    outs, pairs, place, a, b, c = [], [], {}, 0, 0, 0
    for o, (cols, ks) in enumerate(blocks):
        n = int(np.prod(cols))
        outs.append((c, m, n, m + o))
        c += (m + o) * n
        for kd, key in ks:
            ak = [msize * s for s in _strides(kd, gap)[0]]
            if key is None or (key, kd) not in place:
                place[(key, kd)] = a
                a += msize * _strides(kd, gap)[1] + 1
            bk, ksize = _strides(kd, gap)
            bn = [ksize * s for s in _strides(cols, gap)[0]]
            pairs.append((o, len(rows), len(kd), len(cols), place[(key, kd)], b, _pad(rows), _pad(kd), _pad(cols),
                          _pad(am), _pad(ak), _pad(bk), _pad(bn)))
            b += ksize * _strides(cols, gap)[1] + 1
    g = torch.Generator(device="cuda").manual_seed(seed)
    A, B = (torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in (a, b))
    got = _exec(ctx, outs, pairs, A, B, c, alpha)
    ro = _offsets(rows, am)
    for o, (off, _, n, ld) in enumerate(outs):
        want, bound = (torch.zeros((m, n), dtype=torch.float64, device="cuda") for _ in range(2))
        k = 0
        for q in pairs:
            if q[0] == o:
                x = A[q[4] + ro[:, None] + _offsets(q[7][:q[2]], q[10])[None, :]]
                y = B[q[5] + _offsets(q[7][:q[2]], q[11])[:, None] + _offsets(q[8][:q[3]], q[12])[None, :]]
                want += x @ y
                bound += x.abs() @ y.abs()
                k += x.shape[1]
        at = off + torch.arange(m, device="cuda")[:, None] + ld * torch.arange(n, device="cuda")[None, :]
        assert torch.all((got[at] - alpha * want).abs() <= 2 * max(k, 1) * 2.0 ** -53 * abs(alpha) * bound), (o, k)
        assert torch.all(got[off + ld * torch.arange(n, device="cuda")[:, None] + torch.arange(m, ld, device="cuda")] == 7.0)


FEW, MANY = 148 * 128 + 77, 16 * 148 * 128 + 301  # rows: one tile of 128 per SM, and several tiles per block of threads


def _shared(widths, ks):
    return [((w,), [((k,), i) for i, k in enumerate(ks)]) for w in widths]


@pytest.mark.parametrize("rows", [1, 130, FEW // 2 - 300, FEW // 2 + 300, FEW, MANY])
@pytest.mark.parametrize("widths", [(1,), (4,), (3, 2), (8,), (9,), (7, 9), (7, 10), (20, 12), (17, 17, 9)])
def test_rows_and_columns(ctx, rows, widths):
    """A thread per row (4, 8, 16 columns) and fragments of 8 and 32 rows, one chunk and several; k of several buffers."""
    _check(ctx, (rows,), _shared(widths, (14, 5, 16, 2)), alpha=-0.5)


@pytest.mark.parametrize("rows", [1000, FEW])
@pytest.mark.parametrize("n", [3, 13, 25])
@pytest.mark.parametrize("ks", [(1,), (15,), (16,), (17,), (64, 1), (64, 64, 64, 64), (3,) * 25, (0, 5, 0), ()])
def test_k(ctx, rows, n, ks):
    """k around the buffers' 16 and 64 and the staged 256; more A blocks than are kept in shared memory; no k."""
    _check(ctx, (rows,), _shared((n,), ks))


@pytest.mark.parametrize("rows,n,ks", [(FEW, 2, (64,) * 5), (FEW, 7, (64,) * 25), (FEW, 8, (61,) * 26),
                                       (2 * FEW, 5, (64,) * 49), (2 * FEW, 16, (6,) * 140), (2 * FEW, 11, (20,) * 40),
                                       (900, 5, (64,) * 5), (FEW, 16, (64,) * 5), (FEW, 31, (33,) * 9)])
def test_long_k(ctx, rows, n, ks):
    """More k than fragments take: a thread per row with B staged whole or in segments, and tiles."""
    _check(ctx, (rows,), _shared((n,), ks), alpha=3.0)


@pytest.mark.parametrize("rows", [(7, 5, 11), (40, 30, 33)])
@pytest.mark.parametrize("cols", [(2, 3), (4, 5)])
@pytest.mark.parametrize("gap", [0, 3])
def test_tables(ctx, rows, cols, gap):
    """Modes that do not merge: rows, k (one A entry each, more than 16) and B's both directions through tables."""
    _check(ctx, rows, [(cols, [((3, 6), 0), ((2, 5), 1)]), (cols, [((3, 6), 0), ((2, 5), 1)]), ((3,), [((4,), 0)])],
           gap=gap)
