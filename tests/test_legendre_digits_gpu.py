"""The FP64 Legendre contractions by digit products on the tensor cores, at
the sizes where their tiles and chunks end: 16-row groups and 32-row tiles of
N, 32-value chunks and 128-value blocks of K, 64 field-levels a column tile,
and the smallest plans.  Tolerance: the 1e-13 relative L2 that every FP64
transform of this library holds against the oracle (per field-level here)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# (N, I, J, batch)
SIZES = [(1, 64, 2, 1), (2, 64, 4, 3), (15, 64, 16, 1), (30, 64, 32, 2), (31, 64, 34, 63), (32, 96, 34, 64),
         (33, 96, 62, 65), (62, 128, 66, 2), (65, 192, 128, 129), (127, 256, 130, 3), (128, 384, 256, 2),
         (257, 768, 260, 2), (300, 768, 514, 1), (21, 64, 2200, 2)]


@pytest.mark.parametrize("N,I,J,B", SIZES)
def test_edges_match_oracle(dccm, oracle, synth, N, I, J, B):
    s = synth.spectra(N, B, seed=N)
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, B + 1)  # a batch below the plan's largest
    g, go = plan.inverse(s), oracle.sht_inverse(N, I, J, s)
    f, fo = plan.forward(go), oracle.sht_forward(N, I, J, go)
    assert plan.status() == (0, 0)
    for b in range(B):
        assert rel_l2(g[b], go[b]) <= 1e-13 and rel_l2(f[b], fo[b]) <= 1e-13, b


def test_magnitudes_and_zero_field_levels(dccm, oracle, synth):
    """Scales are per field-level and wavenumber: extreme magnitudes share a
    batch with zeros and ordinary values."""
    N, I, J = 42, 128, 64
    mag = np.array([1e-290, 1e290, 0.0, 1.0, 1e-5, 3e17])
    s = synth.spectra(N, len(mag), seed=2) * mag[:, None]
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, len(mag))
    g, go = plan.inverse(s), oracle.sht_inverse(N, I, J, s)
    f, fo = plan.forward(go), oracle.sht_forward(N, I, J, go)
    for b, x in enumerate(mag):
        if x == 0.0:
            assert not g[b].any() and not f[b].any()
        else:
            assert rel_l2(g[b] / x, go[b] / x) <= 1e-13 and rel_l2(f[b] / x, fo[b] / x) <= 1e-13, x


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_stays_in_its_field_level(dccm, synth, bad):
    N, I, J, B = 21, 64, 32, 3
    s = synth.spectra(N, B, seed=1)
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, B)
    g0 = plan.inverse(s)
    f0 = plan.forward(g0)
    t, h = s.copy(), g0.copy()
    t[1, 40] = bad
    h[1, 5, 7] = bad
    g, f = plan.inverse(t), plan.forward(h)
    for b in (0, 2):
        assert np.array_equal(g[b], g0[b]) and np.array_equal(f[b], f0[b])
    assert not np.isfinite(g[1]).any() and not np.isfinite(f[1].real).any()


def test_expired_wait_reports_timeout_then_recovers(dccm, oracle, synth):
    """The bounded waits' failure path: copies withheld (nothing in flight),
    20 ms limit; then the same plan is correct."""
    N, I, J, B = 42, 128, 64, 3
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, B)
    s = synth.spectra(N, B, seed=3)
    saved = {k: dccm.tune_get(k) for k in ("wait_limit_ms", "tc_withhold_loads")}
    try:
        dccm.tune_set("wait_limit_ms", 20)
        dccm.tune_set("tc_withhold_loads", 1)
        for call, x in ((plan.inverse, s), (plan.forward, np.ones((B, J, I)))):
            with pytest.raises(dccm.DccmError) as e:
                call(x)
            assert e.value.status == -8
    finally:
        for k, v in saved.items():
            dccm.tune_set(k, v)
    assert rel_l2(plan.inverse(s), oracle.sht_inverse(N, I, J, s)) <= 1e-13
    assert plan.status() == (0, 0)
