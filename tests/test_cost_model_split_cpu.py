"""The cost model behind TT_PREC_TF32X3_AUTO against times measured on B200, on the host
through tt_contract_predict (no device needed).

Plans with few output tiles and a long k: the FP64 kernel shares a tile's k range among up
to eight CTAs, so it is the faster form there (measured, us, FP64 / 3xTF32: 64 x 64 with k =
2000 24 / 52; 300 x 100 with 8 pairs of 200 22 / 48; 1400 x 100 with 8 pairs of 200 36 / 51;
40 blocks of 40 x 40 with 20 pairs of 300 114 / 278).  Large plans are faster on the tensor
cores (40 blocks of 1400 x 100, k = 400, 228 / 133; three of 1024 x 1024, k = 2000, 472 /
130).  Predictions within 40 % of what was measured.
"""
import ctypes as C

import pytest

MAXM = 6
FP64, TF32X3, TF32X3_AUTO = 0, 2, 4


class OutBlock(C.Structure):
    _fields_ = [("c_off", C.c_int64), ("m", C.c_int32), ("n", C.c_int32), ("ldc", C.c_int32)]


class BlockPair(C.Structure):
    _fields_ = [("out_block", C.c_int32), ("n_m", C.c_int32), ("n_k", C.c_int32), ("n_n", C.c_int32),
                ("a_off", C.c_int64), ("b_off", C.c_int64),
                ("m_dims", C.c_int32 * MAXM), ("k_dims", C.c_int32 * MAXM), ("n_dims", C.c_int32 * MAXM),
                ("a_m_stride", C.c_int64 * MAXM), ("a_k_stride", C.c_int64 * MAXM),
                ("b_k_stride", C.c_int64 * MAXM), ("b_n_stride", C.c_int64 * MAXM)]


def _predict(blocks):
    import tt_b200
    f = tt_b200.lib.tt_contract_predict
    f.restype = C.c_int
    f.argtypes = [C.POINTER(OutBlock), C.c_int, C.POINTER(BlockPair), C.c_int, C.c_int, C.c_int,
                  C.POINTER(C.c_double), C.POINTER(C.c_double), C.POINTER(C.c_int)]
    outs, pairs = [], []
    c = a = b = 0
    for o, (m, n, ks) in enumerate(blocks):
        outs.append(OutBlock(c, m, n, m))
        c += m * n
        for k in ks:
            p = BlockPair()
            p.out_block, p.n_m, p.n_k, p.n_n, p.a_off, p.b_off = o, 1, 1, 1, a, b
            p.m_dims[0], p.k_dims[0], p.n_dims[0] = m, k, n
            p.a_m_stride[0], p.a_k_stride[0], p.b_k_stride[0], p.b_n_stride[0] = 1, m, 1, k
            pairs.append(p)
            a += m * k
            b += k * n
    us64, ustc, choice = C.c_double(), C.c_double(), C.c_int()
    assert f((OutBlock * len(outs))(*outs), len(outs), (BlockPair * len(pairs))(*pairs), len(pairs), TF32X3_AUTO, 148,
             C.byref(us64), C.byref(ustc), C.byref(choice)) == 0
    return us64.value, ustc.value, choice.value


@pytest.mark.parametrize("count,m,n,ks,us64,ustc,choice", [
    (1, 64, 64, [2000], 24.0, 51.7, FP64), (1, 300, 100, [200] * 8, 22.1, 47.8, FP64),
    (1, 1400, 100, [200] * 8, 36.4, 51.0, FP64), (3, 128, 128, [300] * 20, 62.7, 138.3, FP64),
    (40, 40, 40, [300] * 20, 113.7, 278.0, FP64), (10, 128, 128, [2000], 42.0, 64.1, FP64),
    (40, 1400, 100, [400], 228.3, 133.3, TF32X3), (3, 1024, 1024, [2000], 472.1, 130.4, TF32X3),
    (3, 1400, 100, [300] * 20, 294.9, 215.5, TF32X3)])
def test_choice_and_times(count, m, n, ks, us64, ustc, choice):
    p64, ptc, got = _predict([(m, n, ks)] * count)
    assert got == choice, (p64, ptc)
    assert abs(p64 / us64 - 1.0) <= 0.4 and abs(ptc / ustc - 1.0) <= 0.4, (p64, ptc)


def test_narrow_blocks_stay_fp64():
    for m, ks in ((5000, [64]), (200000, [14] * 4), (1000000, [64] * 4)):
        p64, ptc, got = _predict([(m, 14, ks)] * 3)
        assert got == FP64, (p64, ptc)
