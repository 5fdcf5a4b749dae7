"""The diagnostic sums (log g, volume-averaged radii) where their parts meet.

k_continuum leaves four sums per 256 faces, k_finalize adds 1024 of those at a
time. Against the oracle's serial sums; tolerance as derived in
test_gpu_diagnostics.py (6e-8 in log g).
"""
import numpy as np
import pytest

from lcurve_re_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 256, 766, 3,329, 7,168 faces: whole parts, two faces short of one, one over;
# 454 strips: 262,266 faces, 1,025 parts
@pytest.mark.parametrize("nlat1,nlat2", [(13, 24), (51, 13), (24, 75), (20, 454), (454, 13)])
def test_diagnostic_sums_across_parts(engine_fp64, oracle, nlat1, nlat2):
    m, d = W.model(nlat1f=nlat1, nlat2f=nlat2), W.data(5)
    _, _, _, _, sco = oracle.light_curve(m, d, diagnostics=True)
    out = engine_fp64.light_curve_comp(m, d, diagnostics=True)
    np.testing.assert_allclose(out[4:], sco[3:7], rtol=1e-7)
