"""FP64 analysis of rows that are zero but for a few values.

The scale of a row of the fixed-point FFT comes from its largest value, and
its sums are small where few values are not zero: the resolution left to them
is 2^-51 of that value (1,024 points), so the error of a row's coefficients
is below 0.8 x 2^-51 of their size, and with the Legendre products' and the
results' roundings within 4 x 2^-53, r.m.s. over the rows, as an FP64 transform's.
The reference is a long double transform with the plan's own tables.

Constant rows of the largest value below a power of two give the largest sums.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble
LENGTHS = [64, 96, 128, 192, 256, 384, 512, 768, 1024]


@pytest.mark.parametrize("I", LENGTHS)
def test_few_values(dccm, I):
    N, J, counts, reps = 31, 32, (1, 2, 4, 8, 16), 8
    Jh = J // 2
    plan = dccm.ShtPlan(N if I > 64 else 30, I, J, dccm.SHT_FP64, len(counts) * reps)
    N = plan.N
    P, (_, w) = plan.pnm(), plan.gauss()
    ang = 2 * L("3.14159265358979323846264338327950288") * (np.outer(np.arange(N + 1), np.arange(I)) % I).astype(L) / I
    dft = (np.cos(ang) - 1j * np.sin(ang)).T / I
    rng = np.random.default_rng(I)
    g = np.zeros((len(counts), reps, J, I))
    for a, k in enumerate(counts):
        for r in range(reps):
            g[a, r, Jh + r, rng.choice(I, k, False)] = rng.uniform(0.5, 1.0, k) * rng.choice([-1.0, 1.0], k)
    s = plan.forward(g.reshape(-1, J, I)).reshape(len(counts), reps, -1)
    for a, k in enumerate(counts):
        err = []
        for r in range(reps):
            F = g[a, r, Jh + r].astype(L) @ dft
            n, d, first = 0.0, 0.0, 0
            for m in range(N + 1):
                part = slice(first, first + N + 1 - m)
                first += N + 1 - m
                want = P[part, r].astype(L) * (L(0.5) * w[Jh + r]) * F[m]
                if m == 0:
                    want = want.real
                n += float((np.abs(s[a, r, part] - want) ** 2).sum())
                d += float((np.abs(want) ** 2).sum())
            err.append(n / d)
        assert np.sqrt(np.mean(err)) <= 4 * 2.0 ** -53, (k, np.sqrt(np.mean(err)))


@pytest.mark.parametrize("I", LENGTHS)
def test_constant_rows(dccm, I):
    N, J = 15, 16
    v = np.array([1.0, -1.0]) * np.nextafter(2.0 ** np.arange(-3, 4)[:, None], 0.0)
    v = v.ravel()
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 2 * len(v))
    g = np.zeros((2, len(v), J, I))
    g[:] = v[:, None, None]
    g[1, :, :J // 2] *= -1.0  # odd in latitude
    s = plan.forward(g.reshape(-1, J, I)).reshape(2, len(v), -1)
    assert np.abs(s[0, :, 0] - v).max() <= 1e-15 * 8 and np.abs(s[0, :, 1:]).max() <= 1e-15 * 8
    P, (_, w) = plan.pnm(), plan.gauss()
    odd = (P[1] * w[J // 2:]).sum()  # s_1^0 of the sign of the latitude
    assert (np.abs(s[1, :, 1] - v * odd) <= 1e-14 * np.abs(v)).all()
