"""Accuracy of the FP64 transforms, close enough to see their last digits.

The reference is a long double transform with the plan's own tables, so only
the arithmetic is compared.  Noise-like fields, per field-level, relative L2:
the fixed-point FFT rounds below 2^-53 of a row, its results, the Legendre
operands' products and the results a unit of 2^-53 at most each: 4 x 2^-53.
(The lowest digit levels missing would be 4e-14.)

The rows of test_largest_partial_sums give the FFT's fixed point the largest
partial sums that it can meet; an overflow would be as large as the field.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

L = np.longdouble
TOL = 4 * 2.0 ** -53


def _phases(N, I):
    ang = 2 * L("3.14159265358979323846264338327950288") * (np.outer(np.arange(N + 1), np.arange(I)) % I).astype(L) / I
    return np.cos(ang) + 1j * np.sin(ang)


def _tables(P, N, Jh):
    """Per m the table over all latitudes, south to north, in long double."""
    first = 0
    for m in range(N + 1):
        p = P[first:first + N + 1 - m].astype(L)
        sign = np.where(np.arange(N + 1 - m) % 2, -1.0, 1.0).astype(L)
        yield m, slice(first, first + N + 1 - m), np.concatenate([(p * sign[:, None])[:, ::-1], p], axis=1)
        first += N + 1 - m


def _err(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / (np.abs(b) ** 2).sum()))


@pytest.mark.parametrize("N,I,J", [(21, 64, 32), (31, 96, 48), (42, 128, 64), (85, 256, 128)])
@pytest.mark.parametrize("slope", [0.0, 1.5])
def test_noise(dccm, synth, N, I, J, slope):
    B, Jh = 2, J // 2
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, B)
    P, (_, w) = plan.pnm(), plan.gauss()
    n = np.concatenate([np.arange(m, N + 1) for m in range(N + 1)])
    spec = synth.spectra(N, B, seed=N) * np.maximum(n, 1.0) ** (1.5 - slope)
    e = _phases(N, I)
    F = np.zeros((B, J, N + 1), np.clongdouble)
    for m, k, t in _tables(P, N, Jh):
        F[:, :, m] = spec[:, k].astype(np.clongdouble) @ t
    want = F[:, :, 0].real[:, :, None] + 2 * (F[:, :, 1:] @ e[1:]).real
    grid = plan.inverse(spec)
    for b in range(B):
        assert _err(grid[b].astype(L), want[b]) <= TOL
    G = (grid.astype(L) @ np.conj(e).T) / I
    back = np.zeros((B, plan.ncoef), np.clongdouble)
    for m, k, t in _tables(P, N, Jh):
        back[:, k] = (G[:, :, m] * (0.5 * w).astype(L)) @ t.T
    back[:, :N + 1] = back[:, :N + 1].real
    s = plan.forward(grid)
    for b in range(B):
        assert _err(s[b], back[b]) <= TOL


@pytest.mark.parametrize("N,I", [(31, 64), (47, 96), (63, 128), (95, 192), (127, 256), (191, 384), (255, 512), (383, 768),
                                 (511, 1024)])
def test_largest_partial_sums(dccm, oracle, N, I):
    J = N + 1
    j = np.arange(J)
    m = np.where(j < J // 2, J // 2 - 1 - j, j - J // 2) * 2  # a row pair's wavenumber
    ang = 2 * np.pi * ((m[:, None] * np.arange(I)) % I) / I + 0.1
    g = np.zeros((3, J, I))
    # north sign(cos), south sign(sin): |z| = sqrt(2) in phase with the wave, and
    # the two signs that differ
    g[0] = np.where((j >= J // 2)[:, None], np.sign(np.cos(ang)), np.sign(np.sin(ang)))
    g[1] = -g[0]
    g[2] = np.sign(np.cos(ang)) * np.where(j % 2, 1.0, np.nextafter(2.0, 0.0))[:, None]
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 3)
    s, so = plan.forward(g), oracle.sht_forward(N, I, J, g)
    c = np.ones((3, plan.ncoef), complex)
    c[1] = 1j
    c[2] = np.where(np.arange(plan.ncoef) % 2, -1.0, 1.0) * (1 + 1j)
    c[:, :N + 1] = c[:, :N + 1].real
    x, xo = plan.inverse(c), oracle.sht_inverse(N, I, J, c)
    for b in range(3):
        assert rel_l2(s[b], so[b]) <= 1e-13 and rel_l2(x[b], xo[b]) <= 1e-13, b


@pytest.mark.parametrize("N,I,J,batch", [(341, 1024, 512, 900), (255, 768, 384, 1600)])
def test_several_launches(dccm, cuda, N, I, J, batch):
    """Batches whose operand images take more than the plan's 4 GB go in
    several launches, with the results of small batches bit for bit, in the
    native and in SPML's layout."""
    torch = cuda
    P, Q = dccm.ShtPlan(N, I, J, max_batch=batch), dccm.ShtPlan(N, I, J, max_batch=64)
    gen = torch.Generator(device="cuda").manual_seed(N)

    def new(*shape):
        return torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")

    spec = torch.randn(batch, P.ncoef, 2, dtype=torch.float64, device="cuda", generator=gen)
    grid, back, wa = new(batch, J, I), new(batch, P.ncoef, 2), new(batch, P.nwa)
    P.inverse_dev(spec, grid, batch)
    P.forward_dev(grid, back, batch)
    P.wa_xya_dev(grid, wa, batch)
    for b0 in (0, 64 * (batch // 64 // 2), 64 * (batch // 64 - 1), batch - 64):
        g, s, a = new(64, J, I), new(64, P.ncoef, 2), new(64, P.nwa)
        Q.inverse_dev(spec[b0:b0 + 64], g, 64)
        Q.forward_dev(grid[b0:b0 + 64], s, 64)
        Q.wa_xya_dev(grid[b0:b0 + 64], a, 64)
        assert torch.equal(g, grid[b0:b0 + 64]) and torch.equal(s, back[b0:b0 + 64]) and torch.equal(a, wa[b0:b0 + 64]), b0
    assert torch.isfinite(grid).all() and torch.isfinite(back).all()
    assert P.status()[0] == 0
    torch.cuda.empty_cache()
