"""The eclipse boundaries from their roots (ecl_root.cuh) on the CPU.

The bisections of ingress and egress compare a midpoint with intervals
certified around the boundary's root instead of testing it, where they can.
Every answer must be Roche::fblink's (fblink.cpp:34-104): here each midpoint of
both bisections of every face of real grids is answered by the intervals, by
the single evaluation and by the fused search, and by fblink. On ordinary
binaries the intervals must also decide most midpoints, or they are not worth
finding.
"""
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

from lcurve_re_b200 import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "screen", "root_check.cpp")
EXE = os.path.join(HERE, "screen", "_build", "root_check")


@pytest.fixture(scope="module")
def root_check():
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", EXE, SRC])
    return EXE


def _run(exe, m, star, posn):
    c = m.to_c()
    ecl = 1 - star
    ri = np.radians(c.iangle)
    hdr = struct.pack("8d", c.q, np.cos(ri), np.sin(ri), c.delta_phase,
                      c.spin2 if ecl == 1 else c.spin1, c.r2 if ecl == 1 else c.r1, 0.0,
                      float(ecl))
    blob = hdr + struct.pack("q", posn.shape[0]) + np.ascontiguousarray(posn).tobytes()
    out = subprocess.run([exe], input=blob, capture_output=True, timeout=600)
    vals = [int(v) for v in out.stdout.split()]
    return out.returncode, dict(zip(("hits", "tests", "zone", "evals", "searches", "wrong"), vals))


# most: the certified intervals decide at least this share of the midpoints
@pytest.mark.parametrize("most,over", [
    (0.6, {}), (0.6, dict(iangle=90.0)), (0.6, dict(r1=0.002, iangle=88.0)),
    (0.3, dict(r1=0.005, q=0.1, iangle=80.0)),       # grazing
    (0.5, dict(q=0.15, r1=0.012, r2=-1.0, iangle=84.0)),  # lobe-filling donor
    (0.0, dict(q=0.8, r1=-1.0, r2=-1.0, iangle=75.0)),    # both lobes filled, in contact
    (0.6, dict(q=3.0, r2=0.35)), (0.6, dict(spin1=0.0, spin2=0.0)),
    (0.6, dict(spin1=20.0, spin2=1.8, r2=0.15)),
    (0.6, dict(delta_phase="1e-9")), (0.3, dict(delta_phase="1e-4"))])
def test_roots_keep_every_decision(root_check, oracle, most, over):
    m = W.model(nlat1f=16, nlat2f=36, **over)
    tests = zone = 0
    for star in (0, 1):
        rc, r = _run(root_check, m, star, oracle.star_grid(m, star)["posn"])
        assert rc == 0 and r["wrong"] == 0, (star, r)
        tests += r["tests"]
        zone += r["zone"]
    assert tests > 1000
    assert zone >= most * tests, (zone, tests)


# small eclipsers and coarse bisections, where the chord through the reference sphere
# falls to the search's accuracy before the potential reaches its root
@pytest.mark.parametrize("star,over", [
    (0, dict(q=0.0428, iangle=83.0, r1=0.17, r2=0.0634, spin1=7.12, delta_phase="7.5e-5")),
    (1, dict(q=0.794, iangle=83.02, r1=0.087, r2=-1.0, delta_phase="4.64e-5")),
    (1, dict(q=0.313, iangle=89.4, r1=0.00694, r2=-1.0, spin2=0.484, delta_phase="2.49e-6")),
    (1, dict(q=2.76, iangle=79.39, r1=0.01026, r2=0.2134, spin1=14.8, delta_phase="1.12e-6")),
    (1, dict(q=0.705, iangle=83.46, r1=0.0983, r2=0.1346, delta_phase="2.58e-5"))])
def test_short_chords_keep_every_decision(root_check, oracle, star, over):
    m = W.model(nlat1f=20, nlat2f=34, **over)
    rc, r = _run(root_check, m, star, oracle.star_grid(m, star)["posn"])
    assert rc == 0 and r["wrong"] == 0, r
    assert r["tests"] > 100


# the search's second step from less than half of its accuracy to several times it:
# smaller and larger eclipsers, finer and coarser bisections
@pytest.mark.parametrize("r2", [0.08, 0.13, 0.17, 0.19, 0.205, 0.22, 0.235])
@pytest.mark.parametrize("delta", ["1e-6", "1e-7", "1e-8"])
def test_narrowed_gaps_keep_every_decision(root_check, oracle, r2, delta):
    m = W.model(nlat1f=14, nlat2f=20, r2=r2, delta_phase=delta, iangle=87.0)
    rc, r = _run(root_check, m, 0, oracle.star_grid(m, 0)["posn"])
    assert rc == 0 and r["wrong"] == 0, r
    if delta == "1e-7":
        assert r["searches"] <= 0.01 * r["tests"], r


@pytest.mark.parametrize("q,spin,radius", [
    (0.25, 1.0, 0.015), (0.25, 1.0, 0.2), (0.05, 1.0, 0.2), (0.15, 1.0, -1.0), (0.8, 1.0, -1.0),
    (3.0, 1.0, 0.35), (0.25, 0.0, 0.25), (0.25, 3.0, 0.1), (0.01, 1.0, 0.002), (0.9, 1.5, 0.3)])
@pytest.mark.parametrize("acc", [1e-8, 1e-5, 1e-12])
def test_radii_are_the_plain_walks(q, spin, radius, acc):
    """face_chop_root against face_chop, bit for bit, both stars."""
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = os.path.join(HERE, "screen", "_build", "chop_check")
    src = os.path.join(HERE, "screen", "chop_check.cpp")
    hdr = os.path.join(HERE, "..", "lcurve_re_b200", "csrc", "ecl_root.cuh")
    os.makedirs(os.path.dirname(exe), exist_ok=True)
    if not os.path.exists(exe) or os.path.getmtime(exe) < max(os.path.getmtime(src),
                                                              os.path.getmtime(hdr)):
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, src])
    for star in (0, 1):
        out = subprocess.run([exe] + [repr(v) for v in (q, spin, radius, star, acc, 1500)],
                             capture_output=True, timeout=300)
        n, bad = (int(v) for v in out.stdout.split())
        assert n > 30000 and bad == 0 and out.returncode == 0, (star, bad)


# both lobes filled, the mass ratio extreme, the eclipser (large) a slow rotator: the eclipsed
# star digs a well of its own at the near end of the chord, below the lobe's potential
@pytest.mark.parametrize("q", [0.003, 0.02, 0.05, 20.0, 47.0, 300.0])
@pytest.mark.parametrize("spin,iangle,delta", [
    (0.0, 70.0, "1e-8"), (0.0, 90.0, "1e-7"), (0.2, 84.0, "1e-7"), (0.4, 70.0, "1e-7"),
    (0.4, 90.0, "1e-8")])
def test_second_wells_keep_every_decision(root_check, oracle, q, spin, iangle, delta):
    star = 1 if q < 1.0 else 0
    over = dict(nlat1f=16, nlat2f=60, spin1=spin) if star else dict(nlat1f=60, nlat2f=16, spin2=spin)
    m = W.model(q=q, r1=-1.0, r2=-1.0, iangle=iangle, delta_phase=delta, **over)
    rc, r = _run(root_check, m, star, oracle.star_grid(m, star)["posn"])
    assert rc == 0 and r["wrong"] == 0, r
    assert r["tests"] > 10000


# a tiny star 2 as the eclipser: the potential about it carries the rounding of a squared
# distance of order one, 1e-16 over the star's radius cubed
@pytest.mark.parametrize("q", [0.02, 0.3])
@pytest.mark.parametrize("r2", [0.0003, 0.0005, 0.0008, 0.0015])
@pytest.mark.parametrize("r1,iangle,delta", [(0.01, 90.0, "1e-9"), (0.01, 90.0, "1e-7"),
                                             (0.1, 87.4, "1e-9"), (0.1, 87.4, "5e-9")])
def test_tiny_second_stars_keep_every_decision(root_check, oracle, q, r2, r1, iangle, delta):
    m = W.model(q=q, r1=r1, r2=r2, iangle=iangle, delta_phase=delta, nlat1f=120, nlat2f=12)
    rc, r = _run(root_check, m, 0, oracle.star_grid(m, 0)["posn"])
    assert rc == 0 and r["wrong"] == 0, r
    assert r["tests"] > 100


# coarse bisections of contact binaries: the search's accuracy is a good part of the chord, and
# dbrent's way after a halved step hangs on the sign of an exact zero
@pytest.mark.parametrize("q,spin", [(16.9, 1.0), (20.0, 1.0), (47.0, 0.75), (0.0084, 0.9),
                                    (0.0027, 0.75)])
@pytest.mark.parametrize("iangle,delta", [(57.0, "6e-5"), (61.0, "5.3e-5"), (66.0, "4.4e-5"),
                                          (70.0, "6e-5")])
def test_coarse_searches_keep_every_decision(root_check, oracle, q, spin, iangle, delta):
    star = 1 if q < 1.0 else 0
    over = dict(nlat1f=16, nlat2f=90) if star else dict(nlat1f=90, nlat2f=16)
    m = W.model(q=q, r1=-1.0, r2=-1.0, spin1=spin, spin2=spin, iangle=iangle, delta_phase=delta,
                **over)
    rc, r = _run(root_check, m, star, oracle.star_grid(m, star)["posn"])
    assert rc == 0 and r["wrong"] == 0, r
    assert r["tests"] > 10000
