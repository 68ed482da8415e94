"""The Mie bake's kernels at the edges of their tiles: one item, bins off the
angle tile, more than one tile, series of 32 and 33 terms (a warp's), one band
and many shares of radii.  Against the float64 oracle with the tolerances of
test_mie, which hold for averages of 40 radii and more: FP32 angular sums 1e-4,
the FP64 series 1e-9.  (A single sphere's interference minima cancel further
than its FP32 sums resolve; there only the series is checked.)"""

import numpy as np
import pytest

import mie_oracle as mo
from sky_cuda.mie import MieDistribution, bake_phase

pytestmark = pytest.mark.gpu


def _size_parameter(terms: int) -> float:
    """The largest size parameter (to 1e-3) whose series has `terms` terms."""
    x = np.arange(0.5, 60.0, 1e-3)
    n = np.array([mo.mie_terms(v) for v in x])
    return float(x[n == terms][-1])


@pytest.mark.parametrize("terms", [7, 31, 32, 33, 64])
def test_series_around_a_warps_terms(gpu, terms):
    x = _size_parameter(terms)
    r = x * 0.55 / (2.0 * np.pi)
    phase, optics = bake_phase(MieDistribution(r, 1.5, r, r, radii=1), [550.0], [1.5 + 0.01j], bins=65)
    q = mo.efficiencies(1.5 + 0.01j, 2.0 * np.pi / 0.55 * r)
    area = np.pi * r * r
    assert optics["sigma_sca_um2"][0] / area == pytest.approx(q[0], rel=1e-9)
    assert optics["sigma_ext_um2"][0] / area == pytest.approx(q[1], rel=1e-9)
    assert optics["g"][0] == pytest.approx(q[3], rel=1e-9)
    assert phase.shape == (1, 65) and np.all(phase > 0.0)


@pytest.mark.parametrize("bands,radii,bins", [(1, 40, 1), (1, 700, 5), (3, 41, 1023), (2, 47, 1025), (1, 40, 2049),
                                              (33, 45, 64)])
def test_shapes(gpu, bands, radii, bins):
    d = MieDistribution(0.2, 2.0, 0.05, 3.0, radii=radii)
    lam = np.linspace(400.0, 700.0, bands)
    m = np.full(bands, 1.45 + 0.02j)
    phase, optics = bake_phase(d, lam, m, bins=bins)
    assert phase.shape == (bands, bins)
    r, w = mo.lognormal_radii(d.r_mode_um, d.sigma_g, d.r_min_um, d.r_max_um, d.radii)
    for b in {0, bands // 2, bands - 1}:
        want, (sca, ext, g) = mo.size_dist_phase(m[b], lam[b] * 1e-3, r, w, mo.cube_root_mu_grid(bins))
        np.testing.assert_allclose(phase[b], want, rtol=1e-4)
        assert optics["sigma_sca_um2"][b] == pytest.approx(sca, rel=1e-9)
        assert optics["sigma_ext_um2"][b] == pytest.approx(ext, rel=1e-9)
        assert optics["g"][b] == pytest.approx(g, rel=1e-9)
