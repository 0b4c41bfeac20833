"""The Sturm count of the eigensolver's bisection, restated in Python.

The kernel (csrc/tridiag_eig.cu, sturm_count) counts the sign changes of the
leading principal minors of T - x I with T scaled to a norm in [1/2, 1),
off-diagonals floored at 2^-60, no test of a step, and one rescaling every eight
steps, the diagonal padded with 4.  It must give the count of LAPACK's dlaebz
(pivots, a division per step) wherever that is well defined: at probes further
than 1e-9 ||T|| from every eigenvalue, on decaying and clustered spectra, split
blocks (e = 0), zeros of the minors and norms far from 1.
"""
import math

import numpy as np
import pytest
import scipy.linalg as sla

from tests.test_sturm_cpu import DBL_MIN, count_pivot


def count_scaled(d, e, x):
    n = len(d)
    r = np.abs(np.concatenate([e, [0.0]])) + np.abs(np.concatenate([[0.0], e]))
    ex = math.frexp(max(abs(np.min(d - r)), abs(np.max(d + r))))[1]
    ds, es, xs = np.ldexp(d, -ex), np.ldexp(e, -ex), math.ldexp(x, -ex)
    npad = (n + 7) // 8 * 8
    dp = np.concatenate([ds, np.full(npad - n, 4.0)])
    e2 = np.concatenate([[0.0], np.maximum(es * es, 2.0 ** -120), np.zeros(npad - n)])
    pm, p, c = 0.0, 1.0, 0
    for i in range(npad):
        pn = (dp[i] - xs) * p - e2[i] * pm
        c += math.copysign(1.0, pn) != math.copysign(1.0, p)
        pm, p = p, pn
        if i % 8 == 7:
            k = max(math.frexp(p)[1], math.frexp(pm)[1])
            if abs(k) > 300:
                p, pm = math.ldexp(p, -k), math.ldexp(pm, -k)
    return c


def _check(d, e, xs):
    e2 = e * e
    ev = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
    tol = 1e-9 * float(np.abs(ev).max())
    pivmin = DBL_MIN * max(1.0, float(e2.max()) if len(e2) else 1.0)
    r = np.abs(np.concatenate([e, [0.0]])) + np.abs(np.concatenate([[0.0], e]))
    for x in xs:
        if not np.min(d - r) <= x <= np.max(d + r):
            continue  # bisection probes the Gershgorin interval only
        near = int(np.sum(np.abs(ev - x) <= tol))
        assert abs(count_pivot(d, e2, x, pivmin) - count_scaled(d, e, x)) <= near, x


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 64, 150])
@pytest.mark.parametrize("scale", [1.0, 1e6, 1e-9])
def test_decaying_and_clustered_spectra(n, scale):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.exp(-np.linspace(0, np.log(1e14), n)) * rng.uniform(0.5, 1, n)
    lam[: n // 3] = 1e-3
    T, _ = sla.hessenberg((Q * lam) @ Q.T, calc_q=True)
    d, e = scale * np.diag(T), scale * np.diag(T, -1)
    ev = np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1))
    _check(d, e, list(0.5 * (ev[1:] + ev[:-1])) + [0.0, -0.5 * scale, 2.0 * scale] + list(d[:10]))


def test_split_blocks_and_exact_hits():
    rng = np.random.default_rng(2)
    for n in (40, 300):
        d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
        e[rng.integers(0, n - 1, n // 5)] = 0.0
        d[n // 2:] = 0.25          # a long block that is already diagonal, probed at its own value
        e[n // 2:] = 0.0
        ev = np.sort(np.linalg.eigvalsh(np.diag(d) + np.diag(e, 1) + np.diag(e, -1)))
        _check(d, e, list(0.5 * (ev[1:] + ev[:-1])[::7]) + [0.25, 0.0, 0.5] + list(d[:20]))
