"""Sz correlators of a chain longer than the number of sites whose environments go
through it together (64): every entry near the two ends of a group and across them
against the expectation value of the operator's own MPO (mps/observables.cpp:64-103) on
the same state.  Values are at most 1/4 and both sides sum a few hundred products of
numbers of that size: tolerance 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [64, 65, 130])
def test_against_expectation_values(L):
    import tt_b200
    ctx = tt_b200.Context(0)
    try:
        h = np.random.default_rng(L).uniform(-1.0, 1.0, L)
        a = tt_b200.AutoMPO()
        for i in range(L - 1):
            a.add(0.5, "S+", i, "S-", i + 1)
            a.add(0.5, "S-", i, "S+", i + 1)
            a.add(0.7, "Sz", i, "Sz", i + 1)
        for i in range(L):
            a.add(float(h[i]), "Sz", i)
        H = tt_b200.QMPO.from_autompo(a, L)
        psi = tt_b200.QMPS(L, [i % 2 for i in range(L)])
        tt_b200.QDMRG(psi, H).run(2, [8, 8], [1e-12], [3])
        sz, szsz = psi.measure_sz()
        n2 = psi.overlap()
        for i, j in [(0, 1), (0, L - 1), (31, 32), (62, 63), (0, 63), (5, 40), (L - 2, L - 1), (63, 64), (64, 70),
                     (3, 64), (63, 127), (64, 128), (127, 128), (128, 129)]:
            if j >= L:
                continue
            one, two = tt_b200.AutoMPO(), tt_b200.AutoMPO()
            one.add(1.0, "Sz", i)
            two.add(1.0, "Sz", i, "Sz", j)
            assert abs(sz[i] - psi.expectation(tt_b200.QMPO.from_autompo(one, L)) / n2) <= 1e-12, i
            assert abs(szsz[i, j] - psi.expectation(tt_b200.QMPO.from_autompo(two, L)) / n2) <= 1e-12, (i, j)
            assert szsz[j, i] == szsz[i, j]
        assert np.all(np.diag(szsz) == 0.25)
        del psi, H
    finally:
        ctx.close()
