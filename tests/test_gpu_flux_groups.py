"""The fast flux sweep's classes of face groups (dark, bright, signs, ranges).

A warp of the sweep classifies runs and parts of runs by bounds over its own
entries, so the points that share a warp decide which code sums an entry; what
it sums must not depend on it. Time-ordered points give warps narrow arcs of
the orbit (whole groups dark or bright); shuffled, each warp spans it and tests
every element. The two curves must be equal bit for bit, point by point.
"""
import numpy as np
import pytest

from lcurve_re_b200 import workloads as W
from lcurve_re_b200.engine import Engine

pytestmark = pytest.mark.gpu

ECLIPSE = dict(lo=-0.03, hi=0.03)


# sizes at the edges of pairs, parts of 16, runs of 64 and chunks; a tiny star
# whose points all lie around its eclipse; an opaque disc (several-range faces)
@pytest.mark.parametrize("over,npts,span", [
    (dict(nlat1f=9, nlat2f=20), 1, {}), (dict(nlat1f=9, nlat2f=20), 33, {}),
    (dict(nlat1f=40, nlat2f=81), 1000, {}), (dict(nlat1f=17, nlat2f=161), 2411, {}),
    (dict(nlat1f=60, nlat2f=40, limb2="Poly"), 4097, {}),
    (dict(nlat1f=120, nlat2f=50, r1=0.004), 3000, ECLIPSE),
    (dict(nlat1f=80, nlat2f=60, iangle=79.0), 1500, ECLIPSE)])
def test_sums_do_not_depend_on_the_warp(over, npts, span):
    m = W.model(**over)
    d = W.data(npts, **span)
    perm = np.random.default_rng(npts).permutation(npts)
    with Engine(precision="mixed") as e:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
        b = e.light_curve_comp(m, d[perm], scale=False, rdata=False, diagnostics=False)[0]
        np.testing.assert_array_equal(a[perm], b)
        e.set_data(d)
        a = e.light_curve_batch_resident([m, m], scale=False, rdata=False)[0].copy()
        e.set_data(d[perm])
        b = e.light_curve_batch_resident([m, m], scale=False, rdata=False)[0]
        np.testing.assert_array_equal(a[:, perm], b)


def test_opaque_disc_sums_do_not_depend_on_the_warp():
    m = W.cv_disc(nlat1f=40, nlat2f=50, nrad=10, nspot=5)
    d = W.data(700)
    perm = np.random.default_rng(1).permutation(700)
    with Engine(precision="mixed") as e:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
        b = e.light_curve_comp(m, d[perm], scale=False, rdata=False, diagnostics=False)[0]
    np.testing.assert_array_equal(a[perm], b)


# the general sweep: beaming, a limb cut-off, lensing, both laws
@pytest.mark.parametrize("over,npts", [
    (dict(nlat1f=20, nlat2f=41, beam_factor1=1.3, beam_factor2=1.6), 1000),
    (dict(nlat1f=33, nlat2f=90, beam_factor1=1.3, limb2="Poly"), 2500),
    (dict(nlat1f=60, nlat2f=30, mucrit1=0.1, mucrit2=0.2), 700),
    (dict(nlat1f=30, nlat2f=40, glens1=1, roche1=0, eclipse2=0, beam_factor1=1.0), 400),
    (dict(nlat1f=25, nlat2f=31, beam_factor1=1.3, mucrit1=-0.5), 17)])
@pytest.mark.parametrize("span", [{}, ECLIPSE])
def test_general_sums_do_not_depend_on_the_warp(over, npts, span):
    m = W.model(**over)
    d = W.data(npts, **span)
    perm = np.random.default_rng(npts).permutation(npts)
    with Engine(precision="mixed") as e:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
        b = e.light_curve_comp(m, d[perm], scale=False, rdata=False, diagnostics=False)[0]
    np.testing.assert_array_equal(a[perm], b)


# a beamed curve whose chunk of 1024 faces takes 48 KB of shared memory, what a CTA has
# without asking, its barrier aside
def test_general_sweep_at_the_default_shared_memory():
    m = W.model(nlat1f=20, nlat2f=220, beam_factor1=1.3, beam_factor2=1.6)
    d = W.data(12500)
    with Engine(precision="mixed") as e, Engine(precision="fp64") as e64:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
        b = e64.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
    np.testing.assert_allclose(a, b, rtol=1e-5)
