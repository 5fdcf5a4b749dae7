"""The double-precision flux sweep's groups of faces against the oracle, bit for bit.

Groups of 64 and 16 faces are dark, bright or tested face by face by bounds that
the warp holds against its entries; what is skipped must be exact zeros. The
faces lie on a spiral, so that groups are narrow; sizes fall at the edges of
parts, runs and blocks of 1024; ranges and normals include forms that the
bounds cannot hold (ranges outside one turn, normals longer than one).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def flat_grid(n, n0, odd):
    rng = np.random.default_rng(n)
    z = np.linspace(0.999, -0.999, n)
    az = 0.1 * np.sqrt(n) * np.arange(n) / n * 2 * np.pi
    r = np.sqrt(1 - z * z)
    d = np.stack([r * np.cos(az), r * np.sin(az), z])
    ingress = rng.uniform(0.80, 0.999) + 0.01 * rng.random(n)
    ingress = np.where(ingress >= 1, ingress - 1, ingress)
    egress = ingress + rng.uniform(0.02, 0.3) + 0.01 * rng.random(n)
    if odd:
        d[:, rng.random(n) < 0.02] *= 1.5
        k = rng.random(n)
        ingress = np.where(k < 0.02, ingress - 1, np.where(k < 0.04, ingress + 1, ingress))
        egress = np.where(k > 0.98, ingress - 0.1, np.where(k > 0.96, ingress + 1.0, egress))
    p = 0.1 * d * (1 + 0.05 * rng.random(n))
    return dict(dx=d[0], dy=d[1], dz=d[2], px=p[0], py=p[1], pz=p[2],
                flux=rng.uniform(0.5, 1.5, n), n0=n0, in1=ingress[n0:], out1=egress[n0:])


@pytest.mark.parametrize("n,n0,nent,order", [
    (1, 0, 1, "time"), (15, 15, 33, "time"), (63, 16, 1000, "time"), (65, 64, 1023, "shuffled"),
    (1024, 1000, 1024, "time"), (1025, 17, 1300, "shuffled"), (2049, 1024, 8192, "time"),
    (3100, 0, 8300, "time"), (3100, 3100, 2500, "time"), (1500, 700, 130, "one phase")])
@pytest.mark.parametrize("odd", [False, True])
def test_group_classes_leave_the_sums_alone(engine_fp64, oracle, n, n0, nent, order, odd):
    flat = flat_grid(n, n0, odd)
    rng = np.random.default_rng(nent)
    ph = np.linspace(0, 1, nent, endpoint=False) if order != "one phase" else np.full(nent, 0.95)
    if order == "shuffled":
        ph = rng.permutation(ph)
    if order == "time":
        ph[-1] = 1.0  # what a phase just below a whole one is rounded to
    si, ci = np.sin(np.radians(85.0)), np.cos(np.radians(85.0))
    phases = dict(ex=si * np.cos(2 * np.pi * ph), ey=-si * np.sin(2 * np.pi * ph),
                  ez=np.full(nent, ci), phin=ph)
    for star, ltype, kw in ((0, 1, {}), (1, 0, dict(mucrit=0.2)), (0, 0, dict(beam=1.4, mucrit=-0.5)),
                            (1, 1, dict(beam=0.7, glens1=True, rlens1=2e-6)),
                            (1, 1, dict(glens1=True, rlens1=2e-6, mucrit=-0.1))):
        kw = dict(ldc=[0.4, 0.1, 0.05, 0.02], ltype=ltype, spin=1.1, vfac=1e-3, xcofm=0.2, **kw)
        a = oracle.sum_star_multi(star, flat, phases, **kw)
        b = engine_fp64.sum_star_multi(star, flat, phases, **kw)
        np.testing.assert_array_equal(a, b)


# the several-range faces and the disc's elements: points in any order share a warp
# with other ranges and horizons
@pytest.mark.parametrize("npts", [1, 31, 33, 500])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("over", [{}, dict(beam_factor1=1.4, beam_factor2=1.2, mucrit1=-0.3),
                                  dict(iangle=79.0, limb2="Poly")])
def test_disc_sums_do_not_depend_on_the_warp(npts, precision, over):
    from lcurve_re_b200 import workloads as W
    from lcurve_re_b200.engine import Engine
    m = W.cv_disc(nlat1f=30, nlat2f=35, nrad=12, nspot=9, **over)
    d = W.data(npts)
    perm = np.random.default_rng(npts).permutation(npts)
    with Engine(precision=precision) as e:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
        b = e.light_curve_comp(m, d[perm], scale=False, rdata=False, diagnostics=False)[0]
    np.testing.assert_array_equal(a[perm], b)


# a point whose time is not a number spoils no other, whichever lane of a warp it is
@pytest.mark.parametrize("bad", [[16], [1, 16, 33, 48]])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_point_without_a_time_spoils_no_other(bad, precision):
    from lcurve_re_b200 import workloads as W
    from lcurve_re_b200.engine import Engine
    m = W.cv_disc(nlat1f=30, nlat2f=35, nrad=12, nspot=9)
    d = W.data(64)
    with Engine(precision=precision) as e:
        a = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0].copy()
        d["time"][bad] = np.nan
        b = e.light_curve_comp(m, d, scale=False, rdata=False, diagnostics=False)[0]
    rest = np.setdiff1d(np.arange(64), bad)
    np.testing.assert_array_equal(a[rest], b[rest])
    assert np.isnan(b[bad]).all()


# phases outside one turn, as a caller of the face-list sweep may hand them in: the ranges are
# compared with them as they are
@pytest.mark.parametrize("scale,shift", [(1.0, 1.0), (1.0, -1.0), (1.0, 0.5), (3.0, -1.0)])
@pytest.mark.parametrize("n,n0,nent", [(65, 0, 33), (1025, 17, 1300)])
def test_phases_outside_one_turn(engine_fp64, oracle, n, n0, nent, scale, shift):
    flat = flat_grid(n, n0, False)
    ph = scale * np.linspace(0, 1, nent, endpoint=False) + shift
    si, ci = np.sin(np.radians(85.0)), np.cos(np.radians(85.0))
    phases = dict(ex=si * np.cos(2 * np.pi * ph), ey=-si * np.sin(2 * np.pi * ph),
                  ez=np.full(nent, ci), phin=ph)
    kw = dict(ldc=[0.4, 0.1, 0.05, 0.02], ltype=1, spin=1.1, vfac=1e-3, xcofm=0.2)
    for star in (0, 1):
        np.testing.assert_array_equal(oracle.sum_star_multi(star, flat, phases, **kw),
                                      engine_fp64.sum_star_multi(star, flat, phases, **kw))
