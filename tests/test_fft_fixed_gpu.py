"""The FP64 path's fixed-point longitude FFT at every supported length,
against the oracle, on rows where a scale per row pair could go wrong: a
spike, a constant, the Nyquist wave, magnitudes that differ from row to row
by 12 orders, and spectra of one or two coefficients.  Tolerance: the 1e-13
relative L2 of every FP64 transform, per field-level."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (N, I, J): alias-free and linear truncations, odd N, the largest N of a length
SIZES = [(31, 64, 32), (31, 96, 48), (63, 128, 64), (63, 192, 96), (85, 256, 128), (191, 384, 192), (255, 512, 256),
         (300, 768, 320), (511, 1024, 512)]


@pytest.mark.parametrize("N,I,J", SIZES)
def test_forward_rows(dccm, oracle, N, I, J):
    rng = np.random.default_rng(N)
    g = np.zeros((6, J, I))
    g[0, J // 2, 3] = 1.0
    g[1] = 250.0
    g[2] = (-1.0) ** np.arange(I) + 1e-9 * rng.standard_normal((J, I))
    g[3] = rng.standard_normal((J, I)) * 10.0 ** rng.uniform(-6, 6, (J, 1))
    g[4] = 300.0 + 1e-10 * rng.standard_normal((J, I))
    g[5] = rng.standard_normal((J, I))
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 6)
    f, fo = plan.forward(g), oracle.sht_forward(N, I, J, g)
    for b in range(6):
        # the Nyquist wave itself is not represented: its field is compared on its own scale
        ref = np.linalg.norm(fo[b]) if b != 2 else 1.0
        assert np.linalg.norm(f[b] - fo[b]) <= 1e-13 * ref, b


@pytest.mark.parametrize("N,I,J", SIZES)
def test_inverse_rows(dccm, oracle, N, I, J):
    rng = np.random.default_rng(N + 1)
    nc = (N + 1) * (N + 2) // 2
    s = np.zeros((5, nc), complex)
    s[0, 0] = 250.0
    s[1, 0], s[1, nc - 1] = 1.0, 1e-11 + 2e-11j
    s[2, nc - 1] = 1.0 - 1.0j  # n = m = N
    s[3] = rng.standard_normal(nc) + 1j * rng.standard_normal(nc)
    s[4] = s[3] * 10.0 ** rng.uniform(-8, 0, nc)
    s[:, :N + 1] = s[:, :N + 1].real
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 5)
    g, go = plan.inverse(s), oracle.sht_inverse(N, I, J, s)
    for b in range(5):
        assert rel_l2(g[b], go[b]) <= 1e-13, b
