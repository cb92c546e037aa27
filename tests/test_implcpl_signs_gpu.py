"""Implicit-coupling sweeps with factors of either sign and any magnitude.

A row may take the integer arithmetic only if every factor of both its
couplings is positive and ordinary: the diffusion coefficients, the height
differences and the Exner functions of both levels that a half level joins.
The kinds put single negative or extreme factors at the top, inside and at
the bottom of a column, and in single columns of a warp.

The couplings are scaled down so that the mass term dominates every diagonal:
nothing cancels there, so M(k,0) holds 1e-14 relative to itself (some twenty
roundings of 2^-53), while a coupling of the wrong sign moves it by the
square of their ratio, 1e-11 and more.  The other outputs hold the 1e-13 of
every sweep test, of a column's largest finite magnitude (not the coupling
coefficients of the huge couplings, whose own terms cancel to rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MATS = ("UVMtx", "TempMtx", "QMixMtx")
SWEPT = ("DUDt", "DVDt", "DTempDt", "DQMixDt")
COEF = {"v": "VelDiffCoef", "t": "TempDiffCoef", "q": "QMixDiffCoef"}


def _profiles(synth, ncol, kmax, ncmax, kind):
    d = synth.column_profiles(ncol, kmax, ncmax=ncmax, seed=kmax)
    for name in COEF.values():
        d[name] *= 0.1
    some = slice(3, None, 5) if kind.endswith("some") else slice(None)
    kind = kind.split("-")[0]
    if kind == "exner_top":
        d["ExnerFull"][kmax - 1, some] *= -1.0
    elif kind == "exner_top_huge":
        d["ExnerFull"][kmax - 1, some] *= 2.0 ** 120
    elif kind == "exner_mid":
        d["ExnerFull"][kmax // 2, some] *= -1.0
    elif kind == "exner_low":
        d["ExnerFull"][0, some] *= -1.0
    elif kind == "exner_half":
        d["ExnerHalf"][kmax // 2, some] *= -1.0
    elif kind == "coef":
        for name in COEF.values():
            d[name][1 + kmax // 2, some] *= -1.0
    elif kind == "height":  # two levels change places
        d["Height"][kmax // 2:kmax // 2 + 2, some] = d["Height"][kmax // 2:kmax // 2 + 2, some][::-1].copy()
    elif kind == "coef_huge":
        for name in COEF.values():
            d[name][1:kmax, some] *= 2.0 ** 130
    elif kind == "mass_huge":
        d["Press"][:, some] *= 2.0 ** 120
    return d


@pytest.mark.parametrize("ncol,kmax,ncmax", [(70, 4, 1), (45, 9, 2), (33, 2, 3)])
@pytest.mark.parametrize("kind", ["plain", "exner_top", "exner_top-some", "exner_top_huge", "exner_mid", "exner_mid-some",
                                  "exner_low", "exner_half", "coef", "coef-some", "height", "coef_huge", "coef_huge-some",
                                  "mass_huge"])
def test_signs_match_oracle(dccm, oracle, synth, kind, ncol, kmax, ncmax):
    d = _profiles(synth, ncol, kmax, ncmax, kind)
    with np.errstate(all="ignore"):
        o = oracle.implcpl_forward(d, 1, synth.IMPLCPL_CONSTS)
    plan = dccm.ImplCplPlan(ncol, kmax, ncmax, 1, synth.IMPLCPL_CONSTS)
    g = plan.forward(d)
    m = plan.matrices()
    dominated = kind not in ("coef_huge", "coef_huge-some")
    for name in MATS:
        a, b = m[name][1], o[name][1]
        fin = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), fin), name
        if dominated:
            assert (np.abs(a[fin] - b[fin]) <= 1e-14 * np.abs(b[fin])).all(), name

    def same(a, b, name):
        fin = np.isfinite(b)
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isfinite(a), fin), name
        scale = np.max(np.where(fin, np.abs(b), 0.0), axis=-2, keepdims=True)  # a column's
        err = np.abs(np.where(fin, a, 0.0) - np.where(fin, b, 0.0))
        assert (err <= 1e-13 * scale).all(), name

    for name in SWEPT + (("ImplCplCoef1", "ImplCplCoef2") if dominated else ()):
        same(g[name], o[name], name)
    # the backward sweep from the same tendencies, its own matrices
    rng = np.random.default_rng(1)
    for name in SWEPT:
        g[name][..., 0, :] = rng.normal(0.0, 1e-3, g[name][..., 0, :].shape)
    with np.errstate(all="ignore"):
        ob = oracle.implcpl_backward(m, g, synth.IMPLCPL_CONSTS[3])
    hb = {name: np.ascontiguousarray(g[name]) for name in SWEPT}
    plan.backward(hb)
    for name in SWEPT:
        same(hb[name], ob[name], "backward " + name)
