"""FP64 transforms whose results lie at powers of two.

The sums of the digit products are 64-bit integers that are shifted up to the
room they have, before the lowest digits are added: a sum just below a power
of two must not run over.  Every spherical harmonic of a truncation by itself,
with powers of two and their neighbours as coefficients, there and back:
coefficients to 1e-13 of the one that is not zero.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,I,J", [(21, 64, 32), (21, 96, 48), (31, 64, 34), (42, 128, 64)])
@pytest.mark.parametrize("value", [1.0, -1.0, 0.5, 2.0 ** 0.5, np.nextafter(1.0, 0.0), 1j])
def test_single_harmonics(dccm, N, I, J, value):
    nc = (N + 1) * (N + 2) // 2
    s = np.eye(nc) * value + 0j
    if isinstance(value, complex):
        s[:, :N + 1] = 0.0
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, nc)
    back = plan.forward(plan.inverse(s))
    assert np.abs(back - s).max() <= 1e-13


@pytest.mark.parametrize("N,I,J", [(21, 64, 32), (85, 256, 128), (300, 768, 514)])
def test_constant_fields(dccm, N, I, J):
    v = np.concatenate([2.0 ** np.arange(-8, 9), np.nextafter(2.0 ** np.arange(-8, 9), 0.0), -(2.0 ** np.arange(-8, 9)),
                        np.arange(1.0, 14.0)])
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, len(v))
    s = plan.forward(np.ones((len(v), J, I)) * v[:, None, None])
    s[:, 0] -= v
    assert (np.abs(s) <= 1e-13 * np.abs(v)[:, None]).all()
