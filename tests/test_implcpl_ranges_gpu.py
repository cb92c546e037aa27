"""The implicit-coupling sweeps where rows change between the integer
arithmetic and the FP64 form: zero, negative and extreme couplings inside a
column and in single columns of a warp, against the oracle.  Tolerance: the
1e-13 of every sweep test, per array, of its largest finite magnitude; the
same infinities (with sign) and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("DUDt", "DVDt", "DTempDt", "DQMixDt", "ImplCplCoef1", "ImplCplCoef2")


def _same(a, o, name):
    fin = np.isfinite(o)
    assert np.array_equal(np.isnan(a), np.isnan(o)) and np.array_equal(np.isfinite(a), fin), name
    assert np.array_equal(np.sign(a[np.isinf(o)]), np.sign(o[np.isinf(o)])), name
    if fin.any():
        assert np.abs(a[fin] - o[fin]).max() <= 1e-13 * np.abs(o[fin]).max(), name


@pytest.mark.parametrize("kind", ["plain", "zero", "mixed", "tiny"])
@pytest.mark.parametrize("ncol,kmax,ncmax", [(45, 2, 1), (130, 3, 2), (77, 17, 1)])
def test_rows_match_oracle(dccm, oracle, synth, kind, ncol, kmax, ncmax):
    d = synth.column_profiles(ncol, kmax, ncmax=ncmax, seed=5)
    rng = np.random.default_rng(kmax)
    for name in ("VelDiffCoef", "TempDiffCoef", "QMixDiffCoef"):
        k = d[name]
        if kind == "zero" and kmax > 2:  # no diffusion above the lowest layers
            k[kmax // 2 + 1:kmax] = 0.0
        elif kind == "mixed":  # single columns of a warp
            k[:, 3::11] = 0.0
        elif kind == "tiny":  # both sides of 2^-100
            k *= 2.0 ** rng.choice([-110.0, -90.0, 0.0], ncol)
    with np.errstate(all="ignore"):
        o = oracle.implcpl_forward(d, 1, synth.IMPLCPL_CONSTS)
    plan = dccm.ImplCplPlan(ncol, kmax, ncmax, 1, synth.IMPLCPL_CONSTS)
    g = plan.forward(d)
    for c in range(ncol):  # per column: the kinds differ by orders of magnitude
        for name in NAMES:
            _same(g[name][..., c], o[name][..., c], (name, c))
    lev1 = rng.normal(0, 1e-3, (4, ncol))
    for t in (g, o):
        for i, name in enumerate(("DUDt", "DVDt", "DTempDt")):
            t[name][0] = lev1[i]
        t["DQMixDt"][:, 0] = lev1[3]
    with np.errstate(all="ignore"):
        ob = oracle.implcpl_backward(o, o, synth.IMPLCPL_CONSTS[3])
    hb = {name: np.ascontiguousarray(g[name]) for name in NAMES[:4]}
    plan.backward(hb)
    if kind == "plain":
        for name in NAMES[:4]:
            _same(hb[name], ob[name], name)
