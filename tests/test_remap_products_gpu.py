"""Remap products on the integer and the FP64 pipes: both round as IEEE does.

Weights and values of every kind (random bit patterns, neighbours of powers
of two, exact ties, subnormal and overflowing products, zeros of both signs,
infinities and NaN), rows long enough that every product of a row and field
falls on either pipe.  The expected sums are numpy's products and sums in
table order, compared bit for bit (NaN by position).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(rng, n, kind):
    if kind == "bits":
        return rng.integers(0, 2**64, n, dtype=np.uint64).view(np.float64)
    if kind == "ties":  # 27-bit mantissas: products of 54 bits, half of them ties
        return (rng.integers(2**26, 2**27, n) | 1).astype(np.float64) * 2.0 ** rng.integers(-60, 60, n)
    if kind == "edges":
        v = 2.0 ** rng.integers(-540, 540, n)
        return np.nextafter(v, rng.choice([0.0, np.inf], n)) * rng.choice([-1.0, 1.0], n)
    if kind == "special":
        return rng.choice([0.0, -0.0, 5e-324, -2.2e-308, 1.7e308, 1.0, -1.5, 1e-200, np.inf, -np.inf, np.nan], n)
    return rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 6, n)


@pytest.mark.parametrize("fields", [1, 2, 3, 4, 6, 7])
@pytest.mark.parametrize("kind", ["plain", "bits", "ties", "edges", "special"])
def test_products_bit_exact(dccm, cuda, kind, fields):
    torch = cuda
    rng = np.random.default_rng(fields)
    ns, nr = 500, 257
    per = rng.integers(1, 12, nr)
    recv = np.repeat(np.arange(1, nr + 1), per)
    send = rng.integers(1, ns + 1, recv.size)
    coef = _values(rng, recv.size, kind)
    src = _values(rng, ns * fields, kind).reshape(fields, ns)
    with np.errstate(all="ignore"):
        want = np.zeros((fields, nr))
        for r, s, w in zip(recv - 1, send - 1, coef):
            want[:, r] = want[:, r] + src[:, s] * w
    plan = dccm.RemapPlan(ns, nr, send, recv, coef)
    d = torch.from_numpy(src).cuda()
    out = torch.full((fields, nr), 7.0, dtype=torch.float64, device="cuda")
    plan.apply_dev(d, ns, out, nr, fields)
    got = out.cpu().numpy()
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint64)[~nan], want.view(np.uint64)[~nan])
