"""The eclipse stage's kernels against the plain bisection, bit for bit.

A grid of up to 256 faces per SM solves its eclipses in one kernel, a larger one
through a candidate queue in three; both find the boundaries from their roots.
eclipse_warp asks for the plain bisection with Roche::fblink, a warp per face.
All must agree exactly: flags, ingress and egress.
"""
import numpy as np
import pytest

from lcurve_re_b200 import workloads as W
from lcurve_re_b200.engine import Engine

pytestmark = pytest.mark.gpu


# 172 strips: 37,667 faces, 173: 38,106, either side of 148 x 256
@pytest.mark.parametrize("over", [
    dict(nlat1f=5, nlat2f=7), dict(nlat1f=31, nlat2f=64), dict(nlat1f=172, nlat2f=173),
    dict(nlat1f=173, nlat2f=172, r1=0.004, iangle=80.0),
    dict(nlat1f=180, nlat2f=190, q=0.15, r2=-1.0, iangle=80.0),
    dict(nlat1f=40, nlat2f=50, roche1=0), dict(nlat1f=40, nlat2f=50, eclipse2=0)])
def test_eclipse_kernels_agree(over):
    m = W.model(**over)
    with Engine(precision="fp64", eclipse_warp=1 << 30) as plain, Engine(precision="mixed") as e:
        for star in (0, 1):
            a, b = plain.star_grid(m, star), e.star_grid(m, star)
            for k in ("posn", "neclipse", "ecl_in", "ecl_out"):
                np.testing.assert_array_equal(a[k], b[k], err_msg="%s of star %d" % (k, star))
