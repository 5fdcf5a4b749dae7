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


# both lobes filled: second wells on the chords, searches that rounding decides
@pytest.mark.parametrize("star,over", [
    (1, dict(q=0.003, spin1=0.0, iangle=70.0, delta_phase="1e-8")),
    (1, dict(q=0.05, spin1=0.2, iangle=84.0)), (0, dict(q=300.0, spin2=0.0, iangle=90.0)),
    (0, dict(q=20.0, iangle=57.0, delta_phase="6e-5")),
    (1, dict(q=0.0084, spin1=0.9, spin2=0.9, iangle=61.0, delta_phase="5.3e-5"))])
@pytest.mark.parametrize("nlat", [120, 200])
def test_contact_eclipses_agree(star, over, nlat):
    m = W.model(r1=-1.0, r2=-1.0, nlat1f=16 if star else nlat, nlat2f=nlat if star else 16, **over)
    with Engine(precision="fp64", eclipse_warp=1 << 30) as plain, Engine(precision="mixed") as e:
        a, b = plain.star_grid(m, star), e.star_grid(m, star)
        for k in ("neclipse", "ecl_in", "ecl_out"):
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
