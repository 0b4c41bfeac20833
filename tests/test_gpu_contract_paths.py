"""FP64 contractions through the C ABI at the edges of the kernels' tiles.

``tt_contract_plan`` / ``tt_contract_exec`` (the inner loop of qtensor::operator*,
qtensor/qtensor.cpp:652-726) on single contractions chosen to reach every route
of the FP64 path: output blocks around the 64x64 tile and its 16-row and
8-column parts, k around the 16-wide chunk, operands contiguous along either
index, index modes that do not merge into one stride (offset tables), output
blocks without pairs, more pairs than are staged at a time, k ranges long
enough to be shared by a cluster, and the narrow blocks of the bandwidth-bound
path.  Reference: numpy in FP64 on the same strided views; an element that sums
K products may differ by the rounding of two summation orders, at most
2 K 2^-53 sum |a b|.
"""
import ctypes as C
import math

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


def _modes(n, cut):
    """n as two modes when `cut` divides it properly, else one."""
    return [cut, n // cut] if 1 < cut < n and n % cut == 0 else [n]


class Case:
    def __init__(self, rng):
        self.rng, self.outs, self.pairs, self.a, self.b, self.c = rng, [], [], 0, 0, 0

    def out(self, m, n, pad=0):
        self.outs.append((self.c, m, n, m + pad))
        self.c += (m + pad) * n
        return len(self.outs) - 1

    def pair(self, o, k, a_kfast, b_kfast, cuts=(0, 0, 0), gap=0, share_a=None):
        """One pair of output block o: each operand stored with its k modes (kfast) or its rows / columns first,
        `gap` unused elements after the first mode of each dimension so that two modes do not merge."""
        m, n = self.outs[o][1], self.outs[o][2]
        md, kd, nd = _modes(m, cuts[0]), _modes(k, cuts[1]), _modes(n, cuts[2])

        def place(first, second):
            run, out = 1, []
            for dims in (first, second):
                st = []
                for i, d in enumerate(dims):
                    st.append(run)
                    run = run * d + (gap if i == 0 and len(dims) > 1 else 0)
                out.append(st)
            return out, run
        (ak, am), asz = place(kd, md) if a_kfast else [x if i else x[::-1] for i, x in enumerate(place(md, kd))]
        (bk, bn), bsz = place(kd, nd) if b_kfast else [x if i else x[::-1] for i, x in enumerate(place(nd, kd))]
        pad = lambda v: v + [0] * (MAXM - len(v))  # noqa: E731
        a_off = self.a if share_a is None else share_a
        self.pairs.append((o, len(md), len(kd), len(nd), a_off, self.b, pad(md), pad(kd), pad(nd), pad(am), pad(ak),
                           pad(bk), pad(bn)))
        if share_a is None:
            self.a += asz + 1  # odd offsets: blocks are only 8-byte aligned
        self.b += bsz + 1
        return a_off

    def check(self, ctx, alpha=1.0):
        import torch
        import tt_b200
        lib = tt_b200.lib
        lib.tt_contract_plan.restype = lib.tt_contract_exec.restype = C.c_int
        lib.tt_contract_plan.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int,
                                         C.POINTER(C.c_void_p)]
        lib.tt_contract_exec.argtypes = [C.c_void_p] * 5 + [C.c_double]
        lib.tt_plan_destroy.argtypes = [C.c_void_p] * 2
        A, B = self.rng.standard_normal(self.a + 1), self.rng.standard_normal(self.b + 1)
        want, bound = np.full(self.c + 1, 7.0), np.zeros(self.c + 1)
        for off, m, n, ld in self.outs:
            for j in range(n):
                want[off + ld * j:off + ld * j + m] = 0.0
        K = np.zeros(len(self.outs))
        for p in self.pairs:
            K[p[0]] += math.prod(p[7][:p[2]])
        for o, nm, nk, nn, ao, bo, md, kd, nd, am, ak, bk, bn in self.pairs:
            def offs(dims, st, cnt):
                r = np.zeros(1, dtype=np.int64)
                for d, s in zip(dims[:cnt], st[:cnt]):
                    r = (r[None, :] + (np.arange(d) * s)[:, None]).ravel()
                return r
            a = A[ao + offs(md, am, nm)[:, None] + offs(kd, ak, nk)[None, :]]
            b = B[bo + offs(kd, bk, nk)[:, None] + offs(nd, bn, nn)[None, :]]
            off, m, n, ld = self.outs[o]
            at = off + np.arange(m)[:, None] + ld * np.arange(n)[None, :]
            want[at] += alpha * (a @ b)
            bound[at] += 2 * max(K[o], 1) * 2.0 ** -53 * abs(alpha) * (abs(a) @ abs(b))
        dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
        dC = torch.full((self.c + 1,), 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        outs, pairs = np.array(self.outs, dtype=OUT), np.array(self.pairs, dtype=PAIR)
        h = C.c_void_p()
        assert lib.tt_contract_plan(ctx.h, outs.ctypes.data, len(outs), pairs.ctypes.data, len(pairs), 0,
                                    C.byref(h)) == 0, lib.tt_get_last_error()
        try:
            for _ in range(2):
                assert lib.tt_contract_exec(ctx.h, h, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), alpha) == 0
            ctx.sync()
        finally:
            lib.tt_plan_destroy(ctx.h, h)
        got = dC.cpu().numpy()
        assert np.all(np.abs(got - want) <= bound), np.max(np.abs(got - want) - bound)


@pytest.mark.parametrize("a_kfast", [False, True])
@pytest.mark.parametrize("b_kfast", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 33, 65), (15, 40, 7), (16, 41, 8), (17, 63, 9), (33, 64, 16), (63, 65, 17),
                                   (64, 64, 64), (65, 129, 33), (130, 35, 100)])
def test_tile_edges(ctx, m, n, k, a_kfast, b_kfast):
    c = Case(np.random.default_rng(m * 1000 + n * 10 + k))
    c.pair(c.out(m, n, pad=3), k, a_kfast, b_kfast)
    c.out(m, n)  # no pairs: zeros
    c.check(ctx, alpha=-0.5)


@pytest.mark.parametrize("a_kfast,b_kfast", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("gap", [0, 5])
def test_two_mode_indices(ctx, a_kfast, b_kfast, gap):
    """Modes that merge into one stride (gap 0) and modes that need the offset tables."""
    c = Case(np.random.default_rng(3))
    o = c.out(96, 70)
    for k in (6, 48, 90):
        c.pair(o, k, a_kfast, b_kfast, cuts=(12, 6, 7), gap=gap)
    c.check(ctx)


def test_many_pairs_and_shared_k(ctx):
    """More pairs per block than one staging batch, of uneven k, and few tiles with long k."""
    c = Case(np.random.default_rng(4))
    o = c.out(70, 66)
    for i in range(37):
        c.pair(o, 1 + (13 * i) % 40, i % 2 == 0, i % 3 == 0)
    long = c.out(20, 40)
    c.pair(long, 3001, True, True)
    c.pair(long, 2, False, False)
    c.check(ctx, alpha=2.0)


@pytest.mark.parametrize("m", [1, 31, 255, 256, 257, 1000])
@pytest.mark.parametrize("widths", [(1,), (3, 1, 1), (8, 6, 6), (17, 15), (32,)])
@pytest.mark.parametrize("gap", [0, 2])
def test_narrow_blocks(ctx, m, widths, gap):
    """Output blocks of at most 32 columns and short k: several blocks fed by the same A blocks, plus one of its own."""
    c = Case(np.random.default_rng(m + 7 * len(widths)))
    rows = 4 * m if gap else m
    shared = None
    for i, w in enumerate(widths):
        o = c.out(rows, w)
        if shared is None:
            shared = [c.pair(o, k, False, True, cuts=(m if gap else 0, 0, 0), gap=gap) for k in (5, 14, 1)]
        else:
            for a, k in zip(shared, (5, 14, 1)):
                c.pair(o, k, False, True, cuts=(m if gap else 0, 0, 0), gap=gap, share_a=a)
    c.check(ctx)


def test_narrow_blocks_separate(ctx):
    """Narrow blocks of different rows linked through one A block of another shape: the per-block form."""
    c = Case(np.random.default_rng(8))
    for m, n, k in ((300, 32, 64), (1, 1, 1), (513, 9, 40)):
        o = c.out(m, n)
        c.pair(o, k, m % 2 == 0, True)
        c.pair(o, 3, False, False)
    c.check(ctx)
