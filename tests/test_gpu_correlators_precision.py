"""The closing product of the Sz correlators is an FP64 inner product.

``set_precision(op=...)`` is the precision of ``operator*``; the number that closes a
contraction (qtensor::contract, mps/observables.cpp:440-447) is in FP64 whatever it is.
Checked on a 12-site state of integers chosen so that everything before that product is
exact in TF32 (integers of at most 11 bits: 20 rows, entries up to 10; sums below 2^24)
and the product itself, a sum above 2^24, is not exact in FP32: ratios of <Sz_i Sz_6> and
<Sz_6> to 1e-13.
"""
import numpy as np
import pytest

from oracle import qdmrg
from oracle.qtensor import to_dense

pytestmark = pytest.mark.gpu
L, MID = 12, 6


def _integer_state(psi, rng):
    """The outer sites place basis states (entries 0 and 1), the two in the middle hold integers up to 10; those of
    a down spin at the right one are 0 or 1, so that its two spins do not cancel in <Sz>."""
    flat = []
    for i in range(L):
        used = {}  # per sector of the larger bond: its states taken so far
        for qn, qi, data in psi.tensor(i).blocks():
            d = np.zeros(data.shape)
            if i in (MID - 1, MID):
                d[:] = rng.integers(1, 11, data.shape) if i < MID or qn[1][0] > 0 else rng.integers(0, 2, data.shape)
            else:
                q = qi[2] if i < MID else qi[0]
                for k in range(min(data.shape[0], data.shape[2])):
                    at = used.get(q, 0)
                    if at < data.shape[2 if i < MID else 0]:
                        d[(k, 0, at) if i < MID else (at, 0, k)] = 1.0
                        used[q] = at + 1
            flat.append(d.reshape(-1, order="F"))
    psi.set_data(np.ascontiguousarray(np.concatenate(flat)))


@pytest.mark.parametrize("op", ["fp64", "tf32", "tf32x3"])
def test_closing_product(op):
    import tt_b200
    ctx = tt_b200.Context(0)
    try:
        h = np.random.default_rng(5).uniform(-1.0, 1.0, L)
        psi = tt_b200.QMPS(L, qdmrg.neel(L))
        tt_b200.QDMRG(psi, tt_b200.QMPO(L, list(h))).run(4, [64], [1e-30], [4])
        _integer_state(psi, np.random.default_rng(1))
        A = [to_dense(psi.tensor(i).to_oracle()) for i in range(L)]
        tt_b200.set_precision(op=op)
        try:
            sz, szsz = psi.measure_sz()
        finally:
            tt_b200.set_precision()
        del psi
    finally:
        ctx.close()
    z = np.array([-0.5, 0.5])
    step = lambda E, T, f: np.einsum("ab,asc,s,bsd->cd", E, T, f, T)  # noqa: E731
    envs = {None: np.ones((1, 1))}
    for i in range(MID):
        nxt = {k: step(E, A[i], np.ones(2)) for k, E in envs.items()}
        nxt[i] = step(envs[None], A[i], z)
        envs = nxt
    R = np.ones((1, 1))
    for i in range(L - 1, MID, -1):
        R = np.einsum("asc,bsd,cd->ab", A[i], A[i], R)
    ZR = np.einsum("asc,s,bsd,cd->ab", A[MID], z, A[MID], R)
    for k, E in list(envs.items()) + [("right", ZR)]:  # 11 bits: integers, half-integers with Sz in them
        E = E if k is None else 2 * E
        assert np.array_equal(E, np.round(E)) and np.abs(E).max() <= 2048
    want = {k: float(np.sum(E * ZR)) for k, E in envs.items()}
    assert np.sum(np.abs(envs[None] * ZR)) > 2.0 ** 24
    ref = max(range(MID), key=lambda k: abs(want[k]))
    for k in range(MID):
        assert abs(szsz[k, MID] / szsz[ref, MID] - want[k] / want[ref]) <= 1e-13, k
    assert abs(sz[MID] / szsz[ref, MID] - want[None] / want[ref]) <= 1e-13
