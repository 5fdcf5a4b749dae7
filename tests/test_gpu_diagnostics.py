"""The diagnostic sums (k_diag: log g and volume-averaged radii) at grid sizes
around its 2048-face blocks, against the oracle's serial sums.

Tolerance: the faces' float areas, gravities and fluxes may differ by 2 float
ulps (2.4e-7 relative) each; their rounding errors are independent, so over the
n >= 100 faces of the smallest grid a sum of positive terms moves by at most
about 3 * 2.4e-7 / sqrt(100) = 7e-8 relative, and log g (in dex) by 0.43 times
twice that, 6e-8, on a value above 1.
"""
import numpy as np
import pytest

from lcurve_re_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 127 faces; 40 gives 2058, ten past one block; 57 gives two whole blocks and a rest
@pytest.mark.parametrize("nlat1,nlat2", [(8, 10), (39, 40), (40, 57), (113, 9)])
def test_diagnostic_sums_across_blocks(engine_mixed, engine_fp64, oracle, nlat1, nlat2):
    m, d = W.model(nlat1f=nlat1, nlat2f=nlat2), W.data(60)
    _, _, _, _, sco = oracle.light_curve(m, d, diagnostics=True)
    out = engine_fp64.light_curve_comp(m, d, diagnostics=True)
    np.testing.assert_allclose(out[4:], sco[3:7], rtol=1e-7)
    # the same geometry in a mixed context; its float fluxes come from FP32
    # intensities (1e-5), which weigh the mean gravity alone
    out = engine_mixed.light_curve_comp(m, d, diagnostics=True)
    np.testing.assert_allclose(out[4:], sco[3:7], rtol=1e-5)
