"""FP64 analysis of fields that are small or zero over most latitudes.

The table's entries of a large zonal wavenumber fall by hundreds of orders of
magnitude towards the poles, and a field's Fourier coefficients need not.  The
coefficients of one wavenumber (and parity) are accurate relative to their
largest product of a Fourier coefficient and a table entry, whatever the other
wavenumbers hold: the reference is a long double sum over the plan's own
tables.

Bound: a row's transform in FP64 accuracy has an error of a few 2^-53 of the
row's r.m.s. over sqrt(I) in every coefficient, which the sums carry on with
the table's magnitudes; 16 of them are allowed, relative to the largest sum
of magnitudes of the (m, parity).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble


def _fields(mu, J, I, rng):
    lat = np.arcsin(mu)
    g = np.zeros((4, J, I))
    g[0, -6:] = rng.standard_normal((6, I))  # a polar cap of noise
    g[1, :3] = rng.standard_normal((3, I)) * 10.0 ** rng.uniform(-8, 8, (3, 1))
    g[2] = np.exp(-((lat - 1.0) / 0.1) ** 2)[:, None] * rng.standard_normal((J, I))  # a band at 57 degrees
    g[2][np.abs(lat - 1.0) > 0.6] = 0.0
    g[3, J // 2 + J // 5] = rng.standard_normal(I)  # one row
    return g


@pytest.mark.parametrize("N,I,J", [(42, 128, 64), (85, 256, 128), (127, 384, 192)])
def test_small_latitudes(dccm, N, I, J):
    rng = np.random.default_rng(N)
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 4)
    P, (mu, w), Jh = plan.pnm(), plan.gauss(), J // 2
    g = _fields(mu, J, I, rng)
    s = plan.forward(g)
    ang = 2 * L("3.14159265358979323846264338327950288") * (np.outer(np.arange(N + 1), np.arange(I)) % I).astype(L) / I
    dft = (np.cos(ang) - 1j * np.sin(ang)).T / I
    first = 0
    F, rms = {}, np.sqrt((g ** 2).mean(axis=2) / I)
    for b in range(4):
        F[b] = np.zeros((J, N + 1), np.clongdouble)
        rows = np.flatnonzero(rms[b])
        F[b][rows] = g[b, rows].astype(L) @ dft
    for m in range(N + 1):
        tab = (0.5 * w[Jh:]).astype(L) * P[first:first + N + 1 - m].astype(L)
        for b in range(4):
            for p in (0, 1):
                t = tab[p::2]
                if not len(t):
                    continue
                fold = F[b][Jh:, m] + (-1) ** p * F[b][:Jh][::-1, m]
                want = t @ fold
                if m == 0:
                    want = want.real
                got = s[b, first + p:first + N + 1 - m:2]
                bound = 16 * 2.0 ** -53 * (np.abs(t) @ (rms[b, Jh:] + rms[b, :Jh][::-1])).max()
                assert (np.abs(got - want) <= bound).all(), (b, m, p, float(np.abs(got - want).max() / bound))
        first += N + 1 - m


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_at_a_pole(dccm, bad):
    """Where the factors are smallest, and beside zeros."""
    N, I, J = 127, 384, 192
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 2)
    g = np.zeros((2, J, I))
    g[0, -1, 3] = bad
    s = plan.forward(g)
    assert not np.isfinite(s[0].real).any() and not s[1].any()
