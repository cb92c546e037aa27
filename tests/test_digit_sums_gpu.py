"""FP64 analysis of data whose digits follow the table's.

Rows constant along the longitude, with values whose first four 9-bit digits
have the magnitude 255 and the signs of the table's fourth to first digits at
that latitude, so that every product of level 5 has one sign: the largest
sums that level can reach.  They are whole numbers, so the result is the exact
sum rounded once: half a unit in its last place, and the products below
level 8 with the operands' last places, 2^-60 of the largest product each.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _digits(x, E):
    q = np.rint(np.ldexp(x, 62 - E)).astype(np.int64)
    out = []
    for _ in range(6):
        d = (q + 256) % 512 - 256
        out.append(d)
        q = (q - d) >> 9
    return [q] + out[::-1]


@pytest.mark.parametrize("N,I,J", [(21, 64, 2200), (20, 64, 512)])
def test_level_five(dccm, N, I, J):
    Jh, rows = J // 2, np.arange(0, N + 1, 2)
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, len(rows))
    _, w = plan.gauss()
    t = (0.5 * w[Jh:]) * plan.pnm()[rows]  # m = 0, even degrees
    factor = np.frexp(np.abs(t).max(axis=0))[1]
    scaled = np.ldexp(t, -factor)
    g = np.zeros((len(rows), J, I))
    for b in range(len(rows)):
        d = _digits(scaled[b], np.frexp(np.abs(scaled[b]).max())[1])
        x = sum(255 * np.where(d[3 - i] < 0, -1.0, 1.0) * 2.0 ** (-9 * i) for i in range(4))
        x = np.ldexp(x, -factor)  # the sum of the two rows' coefficients
        g[b, Jh:] = 0.5 * x[:, None]
        g[b, :Jh] = 0.5 * x[::-1, None]
    s = plan.forward(g)
    for b in range(len(rows)):
        x = 2 * g[b, Jh:, 0]
        big = Fraction(float(np.abs(np.ldexp(x, factor)).max())) * Fraction(float(np.abs(scaled).max()))
        for k, n in enumerate(rows):
            want = sum((Fraction(float(a)) * Fraction(float(c)) for a, c in zip(x, t[k])), Fraction(0))
            got = Fraction(float(s[b, n].real))
            ulp = Fraction(float(np.spacing(abs(float(want)))))
            assert abs(got - want) <= ulp * Fraction(513, 1024) + Jh * big / 2 ** 60, (b, n, float((got - want) / big * 2 ** 43))
