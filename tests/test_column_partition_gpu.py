"""A column's results do not depend on the columns beside it.

The column physics has two forms of a row (implicit coupling), by the ranges
of that column's own inputs: the same columns in
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
