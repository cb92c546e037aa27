"""The bulk flux on both forms of its column, against the oracle: inputs
inside the integer path's ranges, across their edges (columns of one warp on
either side), and outside.  Tolerance: the 1e-13 relative L2 per output of
every flux test."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

NX, NY = 75, 9  # ragged against warps and CTAs


def _state(synth, kind):
    rng = np.random.default_rng(7)
    ice = np.where(rng.uniform(size=(NX, NY)) < 0.3, rng.uniform(0, 1, (NX, NY)), 0.0)
    d, grid = synth.surface_state(np.linspace(-1.5, 1.5, NY), NX, seed=3, sea_ice=None if kind == "open" else ice,
                                  halo_fill=-1.0)
    it = (slice(1, -1), slice(1, -1))
    d["SfcAirTemp"][it] += rng.normal(0, 3.0, (NX, NY))
    d["ImplCplCoef2"][it] = rng.normal(0, 0.01, (NX, NY, 4))
    if kind == "cold":  # surface temperatures on both sides of 128 K
        d["SfcTemp"][it][..., :2] = rng.uniform(115.0, 141.0, (NX, NY, 2))
        d["SfcAirTemp"][it] = rng.uniform(110.0, 140.0, (NX, NY))
    elif kind == "hot":
        d["SfcTemp"][it][..., :2] = rng.uniform(400.0, 3000.0, (NX, NY, 2))
        d["SfcAirTemp"][it] = rng.uniform(300.0, 2500.0, (NX, NY))
    elif kind == "wind":  # calm to far beyond the upper limit
        s = 10.0 ** rng.uniform(-6, 6, (NX, NY)) * (rng.uniform(size=(NX, NY)) < 0.8)
        d["WindU"][it], d["WindV"][it] = s, -0.3 * s
    elif kind == "pressure":  # any atmosphere, and next to none; the coupling coefficients go with it
        ps = 10.0 ** rng.uniform(-32, 12, (NX, NY))
        d["ImplCplCoef1"][it] *= (ps / d["SfcPress"][it])[..., None]
        d["SfcPress"][it] = ps
    elif kind.startswith("sigma"):
        d["a_Sig1Info"] = np.array([float(kind[5:]), 0.01])
    d.update(synth.flux_outputs(grid[0], grid[1], fill=0.0))
    return d, grid


@pytest.mark.parametrize("kind", ["open", "ice", "cold", "hot", "wind", "pressure", "sigma0.5", "sigma0.99999", "sigma0.9999999"])
def test_ranges_match_oracle(dccm, oracle, synth, kind):
    d, grid = _state(synth, kind)
    ref = {k: v.copy() if v.ndim == 1 else v.copy(order="F") for k, v in d.items()}
    oracle.sfc_bulk_flux(ref, *grid)
    dccm.DSFCM_Util_SfcBulkFlux_Get(d, *grid)
    for n in dccm.FLUX_OUT + ["SfcTemp", "SfcAlbedo"]:
        assert rel_l2(d[n], ref[n]) <= 1e-13, n


@pytest.mark.parametrize("name", ["WindU", "QVap1", "SfcPress", "SfcTemp", "LDwRFlx"])
def test_a_nan_stays_in_its_column(dccm, oracle, synth, name):
    """One NaN input: the column's outputs are NaN where the oracle's are,
    the other columns of its warp are what they were."""
    d, grid = _state(synth, "ice")
    good, ref = ({k: v.copy() if v.ndim == 1 else v.copy(order="F") for k, v in d.items()} for _ in range(2))
    for x in (d, ref):
        x[name][(40, 5) + (0,) * (x[name].ndim - 2)] = np.nan
    oracle.sfc_bulk_flux(ref, *grid)
    dccm.DSFCM_Util_SfcBulkFlux_Get(good, *grid)
    dccm.DSFCM_Util_SfcBulkFlux_Get(d, *grid)
    for n in dccm.FLUX_OUT:
        assert np.array_equal(np.isnan(d[n]), np.isnan(ref[n])), n
        a, b = d[n].copy(), good[n].copy()
        a[40, 5] = b[40, 5] = 0.0
        assert rel_l2(a, b) <= 1e-13, n
