"""FP64 transforms where nearly every operand lies below the last place of the
fixed point: such values round to zero or one unit, not all to one.

One value of 1 among values of +1e-30: the answer is that of the 1 alone to
1e-25, and every product of it is a few correctly rounded operations, so 8
units of 2^-53 of the result's own size are allowed.  Rounded up, the small
ones would add a unit each, which the sums over a row (2^-48 of the mean) and
over all degrees (2^-48 of the value near the poles) show.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 8 * 2.0 ** -53


def test_forward_mean(dccm):
    N, I, J = 20, 1024, 32
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 2)
    _, w = plan.gauss()
    g = np.full((2, J, I), 1e-30)
    g[0, 13, 7] = 1.0
    g[1, 2, 1000] = -1.0
    s = plan.forward(g)
    for b, (j, x) in enumerate(((13, 1.0), (2, -1.0))):
        mean = 0.5 * w[j] * x / I  # s_0^0, Pbar_0^0 = 1
        assert abs(s[b, 0].real - mean) <= TOL * abs(mean), b


def test_inverse_values(dccm):
    N, I, J = 511, 1024, 512
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 2)
    P = plan.pnm()
    s = np.full((2, plan.ncoef), 1e-30 + 1e-30j)
    s[:, :N + 1] = s[:, :N + 1].real
    s[0, 0] = 1.0
    s[1, 10] = 1.0
    g = plan.inverse(s)
    for b, k in enumerate((0, 10)):
        want = np.concatenate([P[k][::-1], P[k]])[:, None]  # even in latitude
        # the sums' unit is 2^-62 of the largest table value times the coefficient
        scale = np.maximum(np.abs(want), 2.0 ** -4 * np.abs(want).max())
        assert (np.abs(g[b] - want) <= TOL * scale).all(), b
