"""A column's results do not depend on the columns beside it.

The column physics has two forms of a column (flux) or row (implicit
coupling), by the ranges of that column's own inputs: the same columns in
another order, or a part of them alone (another domain decomposition), give
the same bits, also where columns of both forms share a warp.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _equal(a, b, name):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    assert np.array_equal(np.isnan(a), np.isnan(b)), name
    ok = ~np.isnan(a)
    assert np.array_equal(a[ok], b[ok]), name


@pytest.mark.parametrize("kind", ["cold", "calm", "ice"])
def test_flux(dccm, synth, kind):
    n = 997
    rng = np.random.default_rng(3)
    ice = np.where(rng.uniform(size=(n, 1)) < 0.3, rng.uniform(0, 1, (n, 1)), 0.0)
    d, grid = synth.surface_state(np.array([0.4]), n, seed=3, sea_ice=None if kind == "calm" else ice, halo_fill=1.0)
    it = (slice(1, -1), slice(1, -1))
    d["ImplCplCoef2"][it] = rng.normal(0, 0.01, (n, 1, 4))
    if kind == "cold":  # surface temperatures on both sides of 128 K, in every warp
        d["SfcTemp"][it][..., :2] = rng.uniform(115.0, 141.0, (n, 1, 2))
        d["SfcAirTemp"][it] = rng.uniform(110.0, 140.0, (n, 1))
    elif kind == "calm":  # winds beyond the range in some columns
        d["WindU"][it] *= np.where(rng.uniform(size=(n, 1)) < 0.1, 2.0 ** 52, 1.0)
    else:
        d["SfcTemp"][it][::7, :, 1] = 100.0  # of ice columns, and of columns without any

    def run(cols):
        m = len(cols)
        x = {"a_Sig1Info": d["a_Sig1Info"]}
        for k, v in d.items():
            if k != "a_Sig1Info":
                x[k] = np.zeros((m + 2,) + v.shape[1:], order="F")
                x[k][1:-1] = v[1:-1][cols]
        x.update(synth.flux_outputs(m + 2, 3, fill=0.0))
        dccm.DSFCM_Util_SfcBulkFlux_Get(x, m + 2, 3, 2, m + 1, 2, 2)
        return {k: x[k][1:-1, 1:-1].copy() for k in dccm.FLUX_OUT + ["SfcTemp", "SfcAlbedo"]}

    whole = run(np.arange(n))
    for cols in [rng.permutation(n), np.arange(5, n, 3)] + [np.array([c]) for c in rng.choice(n, 40, False)]:
        part = run(cols)
        for k, v in part.items():
            _equal(v, whole[k][cols], k)


@pytest.mark.parametrize("kind", ["zero", "tiny", "negative"])
def test_implcpl(dccm, synth, kind):
    n, kmax, nc = 333, 11, 2
    rng = np.random.default_rng(4)
    d = synth.column_profiles(n, kmax, ncmax=nc, seed=4)
    pick = rng.uniform(size=n) < 0.2
    for name in ("VelDiffCoef", "TempDiffCoef", "QMixDiffCoef"):
        f = {"zero": 0.0, "tiny": 2.0 ** -110, "negative": -1e-3}[kind]
        d[name][3:6, pick] *= f
    lev1 = rng.normal(0, 1e-3, (3 + nc, n))

    def run(cols):
        plan = dccm.ImplCplPlan(len(cols), kmax, nc, 1, synth.IMPLCPL_CONSTS)
        out = plan.forward({k: np.ascontiguousarray(v[..., cols]) for k, v in d.items()})
        res = {k: v.copy() for k, v in out.items()}
        res.update({k: v[1].copy() for k, v in plan.matrices().items()})
        t = {k: out[k] for k in ("DUDt", "DVDt", "DTempDt", "DQMixDt")}
        for i, k in enumerate(("DUDt", "DVDt", "DTempDt")):
            t[k][0] = lev1[i, cols]
        t["DQMixDt"][:, 0] = lev1[3:][:, cols]
        plan.backward(t)
        res.update({"backward " + k: v for k, v in t.items()})
        return res

    whole = run(np.arange(n))
    for cols in (rng.permutation(n), np.arange(2, n, 3), np.flatnonzero(pick)[:1], np.flatnonzero(~pick)):
        for k, v in run(cols).items():
            _equal(v, whole[k][..., cols], k)
