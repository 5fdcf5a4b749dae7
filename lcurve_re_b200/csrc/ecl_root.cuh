// ecl_root.cuh — the eclipse boundary of a line of sight from its root.
//
// ingress_egress (ingress_egress.cpp:61-86) bisects the phase at which the
// line of sight to a surface element leaves the eclipsing star: about twenty
// tests Roche::fblink (fblink.cpp:34-104) per boundary, each a search for
// the lowest potential along the chord through the eclipser's reference
// sphere. Almost all of those tests are far enough from the boundary that
// their outcome follows from where the boundary is:
//
//   * fblink's first evaluation is the potential f at the chord's midpoint,
//     the closest approach to the eclipser's centre; f <= pref answers "hidden"
//     at once;
//   * when the lowest potential on the chord exceeds pref, nothing that the
//     search evaluates can reach it: "not hidden" (the lowest on the whole chord,
//     which its minimum near the midpoint need not be, see EdgeEval);
//   * in between, the search's second step answers nearly always (narrow_zone).
//
// edge_zone finds the root of f(phase) - pref by Newton's method and, with a
// bound K on |f''| around it, certifies by Taylor's theorem an interval of
// phases on either side of the root: hidden up to hid, not hidden from vis on
// (vis allows for the depth of the potential's minimum below f). The
// bisection takes the same midpoints as before; inside the certified
// intervals a midpoint is compared instead of tested, and the few between hid
// and vis run fblink. (The eclipser's tide moves the minimum off the midpoint,
// which puts hid and vis about twenty delta_phase apart on an M dwarf before
// narrow_zone, far below one on a white dwarf.) Every decision is fblink's, so
// the phases are the bisection's, bit for bit. eval_edge alone answers the
// midpoints outside the intervals.
//
// All in FP64. Margins cover the rounding of both sides: positions to a few
// ulps of the orbit's size, times the gradient, and the potential itself.
#pragma once

#include "roche.cuh"

namespace lcg {

enum { kEdgeFalse = 0, kEdgeTrue = 1, kEdgeUnsure = 2 };

// Potential about the eclipser's centre (the shift moved into pref):
//   f(u) = -me/|u| - mo/|u - (dx,0,0)| - ss/2 (ux^2 + uy^2) + k ux - pref
// er = me / rref. round: the eclipser's pull exceeds three times what the other terms can
// bend f down by anywhere in the reference sphere (see EdgeEval).
struct EdgeStar {
    double me, mo, dx, ss, k, pref, rref2, cosi, sini, rref, er;
    int32_t round;
};

LCG_HD EdgeStar make_edge_star(int star, double q, double spin, double cosi, double sini,
                               double rref, double pref) {
    EdgeStar s;
    const double mu = q / (1 + q), comp = 1. - mu;
    s.ss = spin * spin;
    if (star == kStar1) {
        s.me = comp; s.mo = mu; s.dx = 1.; s.k = mu;
        s.pref = pref;
    } else {
        // rpot2 = ... - ss (1/2 + (x^2 + y^2) / 2 - x) - comp x with x = 1 + ux
        s.me = mu; s.mo = comp; s.dx = -1.; s.k = -comp;
        s.pref = pref + comp;
    }
    s.rref2 = rref * rref;
    s.rref = rref;
    s.er = s.me / rref;
    const double gap = 1. - rref;  // no point of the sphere is nearer to the other star
    s.round = gap > 0. && s.er / s.rref2 > 3. * (2. * s.mo / (gap * gap * gap) + s.ss);
    s.cosi = cosi;
    s.sini = sini;
    return s;
}

// Whether the chord has no second well. "Not hidden" follows from the potential's minimum
// near the midpoint only where no other lies lower: a contact binary's other star, with
// an extreme mass ratio and the eclipser a slow rotator, digs one at the near end, and
// Roche::fblink finds it. Along the chord f = E + T, the eclipser's term E(t) = -me /
// sqrt(b^2 + t^2), whose slope P(t) = me t / r^3 is at least er3 t, er3 = me / rref^3, and the
// other star's and the rotation's, which bend down by T'' >= -c, c = 2 mo / (1 - rref)^3 + ss.
//   * Round eclipsers, er3 > 3 c, where rref^2 < 1.6 b^2 and the minimum tm lies within b / 9 of
//     the midpoint: past k tm, k = (me / b^3 - c) / (er3 - c) < 2.6, the slope is at least
//     (er3 - c) t - (me / b^3 - c) tm > 0; up to there P' > er3 / 2 > c; on the other side of
//     the midpoint P alone outweighs c. f falls to tm and rises after it: nothing else to see.
//   * Otherwise from a point t1 with f >= f0 and a slope outwards of at least s0 >= 0,
//       f(t) >= M(t) = f0 + E(t) - E(t1) + (s0 - P(t1)) (t - t1) - t2 (t - t1)^2 / 2
//     while T'' >= -t2. M bends down once at most on the way out, so it is lowest at t1 or at
//     the chord's end, where E = -me / rref. Where the chord lies beyond the other star,
//     which the line passes at a distance p, and its near end w beyond that, 2 w^2 >= 3 p^2,
//     T'' falls all the way to the near end: f itself bends down once at most, so its value
//     there decides, and towards the far end t2 is what it is at t1.

// One evaluation on the line of sight at a phase, a distance t beyond the
// chord's midpoint: f, df/dphase (t held), slope g and curvature h along the
// line; squared distances b2 (closest approach), r2 (of the point) from the
// eclipser's centre, distance d from the other star's and its inverse io; x, the
// way to the midpoint, and its rate xp; main term ae = m_e / r^3; a bound tol on
// the rounding of f; the line's direction (ex, ey, cos i).
struct EdgeEval {
    double f, fp, g, h, b2, r2, d, io, x, xp, ae, tol, ex, ey;
    int ans;  // kEdge*: what fblink answers at this phase (t = 0)
    bool on;  // the chord exists and f and the rest are set
};

LCG_HD double edge_rsqrt(double v) {
#ifdef __CUDA_ARCH__
    return rsqrt(v);
#else
    return 1. / sqrt(v);
#endif
}

LCG_HD void edge_sincos(double phase, double &s, double &c) {
#ifdef __CUDA_ARCH__
    sincospi(2. * phase, &s, &c);
#else
    const double r = phase - rint(phase);
    s = sin(kTwoPi * r);
    c = cos(kTwoPi * r);
#endif
}

// u0: the element relative to the eclipser's centre, u2 = |u0|^2; acc: fblink's
// accuracy on the line parameter. An element inside the reference sphere (or
// on it) is left to fblink, which answers "hidden" without a search.
LCG_HD EdgeEval eval_edge(const EdgeStar &S, V3 u0, double u2, double acc, double phase,
                          double t) {
    EdgeEval r;
    r.on = false;
    r.ans = kEdgeUnsure;
    if (!(u2 > S.rref2 * (1. + 1e-9))) return r;
    double sn, cs;
    edge_sincos(phase, sn, cs);
    const double ex = S.sini * cs, ey = -S.sini * sn, ez = S.cosi;
    const double x = -fma(ex, u0.x, fma(ey, u0.y, ez * u0.z));
    const double tiny = 1e-13 * (1. + u2);
    if (x <= tiny) {
        if (x < -tiny) r.ans = kEdgeFalse;  // the eclipser lies behind
        return r;
    }
    const double b2 = u2 - x * x;
    const double hc2 = S.rref2 - b2;  // squared half chord
    const double a2 = 0.25 * acc * acc;
    if (hc2 <= a2 * (1. + 1e-6) + tiny) {
        // no chord, or one no longer than acc: fblink does not search
        if (hc2 < a2 * (1. - 1e-6) - tiny) r.ans = kEdgeFalse;
        return r;
    }
    const double lam = x + t;
    const double ux = fma(lam, ex, u0.x), uy = fma(lam, ey, u0.y), uz = fma(lam, ez, u0.z);
    const double vx = ux - S.dx;
    const double rxy = fma(ux, ux, uy * uy), r2 = fma(uz, uz, rxy);
    const double d2 = fma(vx, vx, fma(uy, uy, uz * uz));
    const double ie = edge_rsqrt(r2), io = edge_rsqrt(d2);
    const double ie2 = ie * ie, io2 = io * io, pe = S.me * ie, po = S.mo * io;
    const double ae = pe * ie2, ao = po * io2;
    r.f = fma(S.k, ux, fma(-0.5 * S.ss, rxy, -(pe + po))) - S.pref;
    const double as = ae + ao - S.ss;
    const double gx = fma(as, ux, fma(-ao, S.dx, S.k)), gy = as * uy, gz = (ae + ao) * uz;
    r.g = fma(gx, ex, fma(gy, ey, gz * ez));
    const double ev = fma(-S.dx, ex, t);  // e.v; e.u = t
    r.h = fma(ae, fma(-3. * t * t, ie2, 1.),
              fma(ao, fma(-3. * ev * ev, io2, 1.), -S.ss * fma(ex, ex, ey * ey)));
    const double px = kTwoPi * ey, py = -kTwoPi * ex;  // de/dphase
    r.xp = -fma(px, u0.x, py * u0.y);
    r.fp = fma(r.xp, r.g, lam * fma(gx, px, gy * py));
    r.b2 = b2;
    r.r2 = r2;
    r.d = d2 * io;
    r.io = io;
    r.x = x;
    r.ex = ex;
    r.ey = ey;
    r.ae = ae;
    // the positions' rounding times the gradients, and that of star 2's squared distance,
    // which Roche::rpot forms as x^2 + y^2 + z^2 + 1 - 2 x (rpot.cpp:37-86)
    r.tol = 1e-14 * (pe * ie + po * io + pe + po + 1.) + 2e-15 * (S.dx < 0. ? ae : ao);
    r.on = true;
    if (r.f <= -r.tol) {
        r.ans = kEdgeTrue;
        return r;
    }
    // the minimum along the chord: at most tau = 2 |g| / h away, where the
    // eclipser's curvature falls by at most 5 (tau / b)^2 of itself (tau <= b / 10)
    // and the other star's changes by at most 6 mo / r^4 per length
    if (r.f > r.tol && r.h > 0.) {
        const double ag = fabs(r.g), tau = 2. * ag / r.h, near = r.d - tau;
        if (100. * tau * tau <= b2 && tau * tau <= hc2 && near > 0.1) {
            const double c3 = 6. * S.mo / (near * near * near * near);
            const double hmin = r.h - 5. * ae * tau * tau * ie2 - c3 * tau;
            const double low = r.f - ag * ag / (2. * hmin);
            if (hmin >= 0.5 * r.h && low > r.tol) {
                if (S.round && S.rref2 < 1.6 * b2) {
                    r.ans = kEdgeFalse;
                } else {
                    // the chord's ends, from tau on, where the slope is at least hmin tau - |g|
                    const double hc = hc2 * edge_rsqrt(hc2), wn = ev - hc, p2 = d2 - ev * ev;
                    const double c = (hmin - ae) * tau - ag, curl = r.h < ae ? ae - r.h : 0.;
                    const double nx = fma(-hc, ex, ux), ny = fma(-hc, ey, uy);
                    const double fn = fma(S.k, nx, fma(-0.5 * S.ss, fma(nx, nx, ny * ny),
                                                       -S.mo * edge_rsqrt(fma(wn, wn, p2)))) -
                                      S.er - S.pref;
                    // (towards the far end it rises from the midpoint on where g > 0)
                    const double up = r.g > 0. ? r.f + ag * hc
                                               : low - 0.5 * ae * tau * tau + (c < 0. ? c : 0.) * hc;
                    const double far = up + pe - S.er - 0.5 * curl * hc2;
                    if (wn > 0. && 2. * wn * wn >= 3. * p2 && fn > r.tol && far > r.tol)
                        r.ans = kEdgeFalse;
                }
            }
        }
    }
    return r;
}

// Roche::fblink's search with one evaluation of value and slope per point
// (both square roots as reciprocals, shared), for the phases between the
// certified intervals: the same chord, bracket check and dbrent
// (dbrent.cpp:21-126) steps, so the same answer except where rounding could
// decide it; there kEdgeUnsure hands the phase to fblink itself: a value within rounding of
// pref or of the one it is compared with, a bracket that fails, and points within mx of
// where dbrent would choose otherwise (far more than a secant step makes of the slopes'
// rounding). That is not rare: after a halved step the best point is the bracket's
// middle, and which way dbrent then moves by acc is the sign of an exact zero. Of the about
// 720 FP64 instructions of an fblink that searches, some 270 remain.
LCG_HD int fblink_edge(const EdgeStar &S, V3 u0, double u2, double acc, double phase) {
    double sn, cs;
    edge_sincos(phase, sn, cs);
    const double ex = S.sini * cs, ey = -S.sini * sn, ez = S.cosi;
    const double B = fma(ex, u0.x, fma(ey, u0.y, ez * u0.z)), C = u2 - S.rref2;
    const double fac = B * B - C, tiny = 1e-12 * (1. + u2);
    if (!(B < -tiny && fac > tiny && C > tiny)) return kEdgeUnsure;
    const double lam2 = sqrt(fac) - B, lam1 = C / lam2, mx = 1e-9 * (lam2 - lam1);
    if (!(lam2 - lam1 > acc * (1. + 1e-9))) return kEdgeUnsure;
    const double exy2 = fma(ex, ex, ey * ey), uxy = fma(ex, u0.x, ey * u0.y);
    double ie = 0., io = 0.;
    auto eval = [&](double l, double &f, double &d) {
        const double ux = fma(l, ex, u0.x), uy = fma(l, ey, u0.y), uz = fma(l, ez, u0.z);
        const double vx = ux - S.dx, yz = fma(uy, uy, uz * uz), eu = l + B;
        ie = edge_rsqrt(fma(ux, ux, yz));
        io = edge_rsqrt(fma(vx, vx, yz));
        const double pe = S.me * ie, po = S.mo * io;
        f = fma(S.k, ux, fma(-0.5 * S.ss, fma(ux, ux, uy * uy), -(pe + po))) - S.pref;
        d = fma(pe * ie * ie, eu,
                fma(po * io * io, fma(-S.dx, ex, eu), fma(-S.ss, fma(l, exy2, uxy), S.k * ex)));
    };
    double x = lam1 + (lam2 - lam1) / 2., fx, dx, f1, f2, t;
    eval(x, fx, dx);
    const double ib = ie;  // the midpoint is the point nearest to the eclipser
    eval(lam2, f2, t);
    const double i2 = io;
    eval(lam1, f1, t);
    // the other star is nearest at an end, unless the line passes it within the chord
    const double in = io > i2 ? io : i2, is = S.dx < 0. ? ib : in;
    if (!(fma(-S.dx, ex, lam1 + B) * fma(-S.dx, ex, lam2 + B) > 0.)) return kEdgeUnsure;
    const double tol = 1e-14 * (S.me * ib * ib + S.mo * in * in + fabs(S.pref) + 10.) +
                       2e-15 * (S.dx < 0. ? S.me : S.mo) * is * is * is;
    if (fabs(fx) <= tol) return kEdgeUnsure;
    if (fx < 0.) return kEdgeTrue;
    // the first level of fblink's subdivision brackets the minimum
    if (!(fx < f1 - tol && fx < f2 - tol)) return kEdgeUnsure;
    double a = lam1, b = lam2, w = x, v = x, fw = fx, fv = fx, dw = dx, dv = dx;
    double e = 0., d = 0.;
    const double tol1 = acc, tol2 = 2. * acc;
#pragma unroll 1
    for (int iter = 0; iter < 100; iter++) {
        const double xm = 0.5 * (a + b), gap = fabs(x - xm) - (tol2 - 0.5 * (b - a));
        if (fabs(gap) <= mx) return kEdgeUnsure;
        if (gap < 0.) return kEdgeFalse;
        bool half = true;
        if (fabs(e) > tol1) {
            double d1 = 2. * (b - a), d2 = d1;
            if (dw != dx) d1 = (w - x) * dx / (dx - dw);
            if (dv != dx) d2 = (v - x) * dx / (dx - dv);
            const double u1 = x + d1, u2_ = x + d2;
            const bool ok1 = (a - u1) * (u1 - b) > 0. && dx * d1 <= 0.;
            const bool ok2 = (a - u2_) * (u2_ - b) > 0. && dx * d2 <= 0.;
            const double olde = e;
            e = d;
            if (ok1 || ok2) {
                const double dn = ok1 && ok2 ? (fabs(d1) < fabs(d2) ? d1 : d2) : ok1 ? d1 : d2;
                const double much = fabs(dn) - fabs(0.5 * olde);
                if (fabs(much) <= mx) return kEdgeUnsure;
                if (much < 0.) {
                    const double u = x + dn, la = u - a, lb = b - u;
                    const double end = (la < lb ? la : lb) - tol2;
                    d = end < 0. ? dsign(tol1, xm - x) : dn;
                    if (fabs(end) <= mx || (end < 0. && fabs(xm - x) <= mx)) return kEdgeUnsure;
                    half = false;
                }
            }
        }
        if (half) d = 0.5 * (e = (dx >= 0. ? a - x : b - x));
        const bool far = fabs(d) >= tol1;
        const double u = far ? x + d : x + dsign(tol1, d);
        double fu, du;
        eval(u, fu, du);
        if (fabs(fu) <= tol || fabs(fu - fx) <= tol) return kEdgeUnsure;
        if (fu < 0.) return kEdgeTrue;
        if (!far && fu > fx) return kEdgeFalse;
        if (fu <= fx) {
            if (u >= x) a = x; else b = x;
            v = w; fv = fw; dv = dw;
            w = x; fw = fx; dw = dx;
            x = u; fx = fu; dx = du;
        } else {
            if (u < x) a = u; else b = u;
            if (fu <= fw || w == x) {
                v = w; fv = fw; dv = dw;
                w = u; fw = fu; dw = du;
            } else if (fu < fv || v == x || v == w) {
                v = u; fv = fu; dv = du;
            }
        }
    }
    return kEdgeUnsure;
}

// Certified phases of one boundary; dir = +1 when the eclipse ends with growing
// phase. fblink answers "hidden" for -hrad <= dir (phase - hc) <= hid and "not
// hidden" for vis <= dir (phase - vc) <= vrad (a radius of 0: nothing).
struct EdgeZone {
    double hc, hrad, hid, vc, vrad, vis;
};

// Bounds within a phase radius rad of the point v was taken at, where the
// point's distance r from the eclipser changes by at most a tenth of itself
// and the one from the other star by no more (P the point on the line):
//   |P'| <= 2 pi (lam + |t|), |P''| <= 4 pi^2 (2 lam + 2 |t| + 2.2 r),
//   |f''| <= |P'|^2 |H| + |P''| |grad f| = K.
// t1, t2 bound the gradient and the second derivatives of the other star's and
// the rotation's terms.
struct EdgeBound {
    double K, t1, t2, rad;
};
LCG_HD EdgeBound edge_bound(const EdgeStar &S, const EdgeEval &v, double lam) {
    EdgeBound B;
    const double r = sqrt(v.r2);
    const double ni = 1.12 * v.io, ni2 = ni * ni;
    B.t1 = S.mo * ni2 + 1.1 * S.ss * r + fabs(S.k);
    B.t2 = 2. * S.mo * ni2 * ni + S.ss;
    const double two2 = kTwoPi * kTwoPi;
    B.K = two2 * (lam * lam * (2.75 * v.ae + B.t2) + (2. * lam + 2.2 * r) * (1.24 * v.ae * r + B.t1));
    const double reach = r * v.io < 1. ? r : 1. / v.io;
    B.rad = 0.1 * reach / (kTwoPi * lam);
    return B;
}

// The part of a phase radius rad around v (edge_zone's stage 1) over which the chord has
// no second well, 0 for none: above, from the minimum, which lies within a of the midpoint
// and is above zero from vis on (vis < 0 reaches inwards of v). For a round eclipser that is
// all of rad, over which b keeps 0.9 of itself. Else, while the chord keeps most of its
// length y, by its far end, where M is above zero if
//   E(y) - E(a) > (me / r^3) a y + t2 (y + a)^2 / 2
// with t2 as it is at the minimum, and by f at the near end, less what it can lose on its
// way. Of lobe-filling donors' boundaries 99.9% are certified so.
LCG_HD double clear_radius(const EdgeStar &S, V3 u0, const EdgeEval &v, double dir, double t,
                           double lam, double dt, double drift, double move, double vis,
                           double rad) {
    const double at = fabs(t), hc2 = S.rref2 - v.b2;
    double a = at + fabs(dt) + drift * rad;
    if (S.round && S.rref2 < 1.3 * v.b2 && 100. * a * a < v.b2) return rad;
    // b^2 grows outwards by 0.8 to 1.2 db2 per phase
    const double db2 = -2. * v.x * v.xp * dir, bend = kTwoPi * kTwoPi / 1.1 * lam * lam;
    if (!(db2 > 0.)) return 0.;
    if (rad * bend > 0.1 * db2) rad = 0.1 * db2 / bend;
    const double in = vis < 0. ? -2.1 * kTwoPi * lam * lam * vis : 0.;
    if (!(in < 0.05 * v.b2 && hc2 > 0.)) return 0.;
    const double ae = 1.15 * v.ae;  // of the minimum, anywhere in the zone
    // the far end: t2 is the other terms' curvature at v, with what it changes by
    const double ih = edge_rsqrt(hc2), hc = hc2 * ih, io2 = v.io * v.io, ib2 = 1. / db2;
    const double t0 = v.ae * (1. - 3. * t * t / v.r2) - v.h;
    const double tv = (t0 > 0. ? t0 : 0.) + 9. * S.mo * io2 * io2 * move;
    double r1 = 0.;
#pragma unroll 1
    for (int i = 0; i < 2; i++) {
        const double keep = i ? 0.92 : 0.75;
        r1 = (1. - keep) / 1.2 * hc2 * ib2;
        if (r1 > rad) r1 = rad;
        a = at + fabs(dt) + drift * r1;
        const double tf = tv + 9. * S.mo * io2 * io2 * a +
                          2. * kTwoPi * r1 * (2.7 * S.mo * io2 * v.io + S.ss);
        const double yl = (i ? 0.9591 : 0.8660) * hc;
        const double ib = edge_rsqrt(S.rref2 - yl * yl + a * a);
        const double ey = S.me * ib - S.er, ey2 = (1. - 3.2 * a * a / v.b2) * S.me * ib * ib * ib;
        // the eclipser's pull at the minimum counts against the end on its own side only
        const double pull = t + (a - at) < 0. ? 0. : ae * a;
        // and from there on, E growing by at least ey2 / 2 per y^2
        if (25. * a * a < v.b2 && ey > pull * yl + 0.5 * tf * (yl + a) * (yl + a) &&
            ey2 * yl > pull + tf * (yl + a))
            break;
        if (i) return 0.;
    }
    const double ex = v.ex, ey = v.ey, ez = S.cosi, l = v.x - hc;
    const double nx = fma(l, ex, u0.x), ny = fma(l, ey, u0.y), nz = fma(l, ez, u0.z);
    const double vx = nx - S.dx, dn2 = fma(vx, vx, fma(ny, ny, nz * nz)), ni = edge_rsqrt(dn2);
    const double wn = fma(ex, vx, fma(ey, ny, ez * nz));
    const double fn = fma(S.k, nx, fma(-0.5 * S.ss, fma(nx, nx, ny * ny), -S.mo * ni)) - S.er - S.pref;
    if (!(wn > 0. && dn2 - wn * wn < 0.22 * dn2 && fn > 0.)) return 0.;
    // the near end's speed along the sphere, and that of the other star's distance; x > hc,
    // the element being outside the sphere
    const double vel = kTwoPi * (lam + 1.) + 1.4 * db2 * ih;
    const double grad = 1.25 * S.mo * ni * ni + fabs(S.k) + 1.1 * S.ss * S.rref;
    const double most = 0.1 * dn2 * ni;
    double r2 = 0.9 * fn;
    if (r2 > most * grad) r2 = most * grad;
    if (r1 * vel * grad > r2) r1 = r2 / (vel * grad);
    if (r1 * (kTwoPi * lam) > 0.1 * v.x) r1 = 0.1 * v.x / (kTwoPi * lam);
    return r1 < -vis ? 0. : r1;
}

// What is known at the visible end of a boundary (edge_zone's stage 1), for
// narrow_zone.
struct EdgeEnd {
    double t, dt, tol;           // offset of the minimum, its last step; rounding of f
    double s0, off, fp, fl, K, rad;  // the Newton root of the minimum, its error, bounds
    double gp, move, t3, vis0;   // bounds; where f(midpoint) > 0 from on, from hc
    double r, h, ae, io, b2, x, ex, ey;  // EdgeEval's
};

// Between hid and vis fblink searches: f > pref at the midpoint x, the minimum
// below. Its dbrent starts at x with slope -g and tries, first, half way to the
// chord's end (u1, always higher: f rises); second, u2 = x + max(d1, acc), d1 the
// secant step from the slopes at x and u1, to within err of the minimum; and third,
// acc to one side of u2. So
//   * u2 = x + acc, f(u2) > f(x) (the minimum is nearer to x than acc / 2): dbrent
//     stops there, "not hidden" wherever f(x) > pref;
//   * u2 = x + acc, f(u2) about f(x) or below: "hidden" where either is below pref;
//     where neither is, dbrent stops there or, after u2 + acc, with the bracket closed;
//   * u2 further, err below about acc / 2: "hidden" where f(u2) < pref, else not. The
//     secant step from u2 is shorter than acc: dbrent moves acc instead and, finding
//     f higher, stops; or, where that ends within 2 acc of x, it tries u2 + acc and if
//     need be u2 - acc, both higher, and the bracket is closed;
//   * otherwise f(u2) <= minimum + 0.7 h err^2, and "hidden" where that is below pref.
// In all but the last the answer turns at the root of f, at x or at u2, and the gap
// between hid and vis shrinks to the error of that root. Over the gap's width om all of
// this moves by bounded amounts; what the bounds leave open is searched as before.
// M-dwarf boundaries on 60-400 strips: 3.3 -> 0.003 searches each.
LCG_HD void narrow_zone(const EdgeStar &S, V3 u0, double acc, double dir, double lam,
                        const EdgeEnd &E, const EdgeBound &B, EdgeZone &z) {
    const double om = 1.05 * (dir * (z.vc - z.hc) - z.hid + fabs(E.s0) + E.off);
    const double hc2 = S.rref2 - E.b2, db = 2. * kTwoPi * lam * lam * om;  // of b^2 and hc^2
    if (!(om > 0. && om < 0.5 * E.rad && om < 0.5 * z.hrad && db < 0.2 * hc2 && hc2 < 0.6 * E.b2))
        return;
    const double hc = sqrt(hc2), dhc = 0.6 * db / hc;
    if (!(hc * E.io < 0.3 && hc > 5. * acc)) return;
    // along the chord the slope grows by rise per length at least, so f has one
    // minimum there, no further than g / rise from the midpoint
    const double ni = E.io / (1. - 1.1 * hc * E.io), ir = edge_rsqrt(S.rref2);
    const double t2 = 2. * S.mo * ni * ni * ni + S.ss, rise = S.me * ir * ir * ir - t2;
    if (!(rise > 0.3 * t2)) return;
    const double ex = E.ex, ey = E.ey, ez = S.cosi, x = E.x;
    const double tm = fabs(E.t + E.dt), sg = E.t + E.dt > 0. ? 1. : -1.;
    // slopes towards the minimum at x (g), u1 (g1) and u2; the value at u2 (f2)
    double g = 0., g1 = 0., d1 = 0., den = 1., step = 0., f2 = 0.;
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
        const double t = i == 0 ? 0. : i == 1 ? 0.5 * sg * hc : sg * step, l = x + t;
        const double ux = fma(l, ex, u0.x), uy = fma(l, ey, u0.y), uz = fma(l, ez, u0.z);
        const double vx = ux - S.dx, yz = fma(uy, uy, uz * uz);
        const double ie = edge_rsqrt(fma(ux, ux, yz)), io = edge_rsqrt(fma(vx, vx, yz));
        const double pe = S.me * ie, po = S.mo * io;
        const double d = sg * fma(pe * ie * ie, t,
                                  fma(po * io * io, fma(-S.dx, ex, t),
                                      fma(-S.ss, fma(ux, ex, uy * ey), S.k * ex)));
        if (i == 0) {
            g = -d;
        } else if (i == 1) {
            g1 = d;
            den = g + g1;
            d1 = 0.5 * hc * g / den;
            step = d1 > acc ? d1 : acc;
        } else {
            f2 = fma(S.k, ux, fma(-0.5 * S.ss, fma(ux, ux, uy * uy), -(pe + po))) - S.pref;
        }
    }
    const double dg = E.gp * om, gmax = g + dg, up = gmax / rise;
    // the slope at u1 moves with the phase and with u1
    const double gp1 = kTwoPi * (2.1 * E.ae * hc / E.r * lam + 2. * (B.t2 * lam + B.t1));
    const double dw = gp1 * om + 0.6 * dhc * (1.3 * E.ae + B.t2);
    if (!(g > 3. * dg && den > 0.25 * rise * hc && 20. * up * up < E.b2 && hc > 5. * up)) return;
    const double rel = dhc / hc + dg / g + (dg + dw) / den;
    if (!(rel < 0.2 && 0.45 * hc - 1.3 * d1 > 2.2 * acc && hc > 4.8 * step)) return;
    const double et = fabs(E.dt) + dg / (0.6 * E.h), du = 1.3 * d1 * rel;
    const double err = fabs(step - tm) + du + et;
    const bool near = acc + tm + et < E.move, one = d1 + du < acc * (1. - 1e-9);
    const double hmin = E.h - E.t3 * (acc + tm + et), far = acc - err;
    const double dh = E.t3 * (1.5 * acc + et), vis0 = dir * (z.hc - z.vc) + E.vis0 + 4e-15;
    if (near && one && 0.5 * hmin * acc > gmax * (1. + 1e-6) + 1e-9) {
        if (vis0 < z.vis) z.vis = vis0;
    } else if (near && (one ? err < 0.6 * acc
                            : err < 0.4 * tm && err < 0.5 * acc &&
                                  far * far * (E.h - dh) > 1.01 * err * err * (E.h + dh))) {
        // df(u2)/dphase: fp at the minimum; the way from there to u2, u2's own motion, K om
        const double e = E.gp * err + 1.4 * E.h * err * du / om + E.K * om;
        const double s2 = f2 / E.fp, off = (fabs(s2) * e + 8. * E.tol) / (E.fp - e) + 8e-15;
        if (!(e < 0.5 * E.fp && fabs(s2) + off < om)) return;
        const double to = dir * (z.vc - z.hc) - s2 - off;
        const double vis = one && vis0 > off - s2 ? vis0 : off - s2;
        if (to > z.hid) z.hid = to;
        if (vis < z.vis) z.vis = vis;
    } else if (err + et < 0.5 * E.move) {
        // f(u2) < pref where the minimum is this deep
        const double del = 1.3 * (E.off + (0.7 * E.h * err * err + 8. * E.tol) / E.fl);
        const double to = dir * (z.vc - z.hc) - E.s0 - del - 8e-15;
        if (E.K * (fabs(E.s0) + del) <= 0.2 * E.fl && fabs(E.s0) + del < E.rad && to > z.hid)
            z.hid = to;
    }
}

// The intervals of one boundary of ingress_egress's bracket: pin the phase
// pot_min found hidden, pout where the line touches the reference sphere;
// delta the bisection's accuracy: intervals that end within a twentieth of it of
// the root are near enough, but narrow_zone's error grows with the distance from the
// minimum's, which one more of Newton's steps makes nothing.
LCG_HD EdgeZone edge_zone(const EdgeStar &S, V3 u0, double acc, double delta, double pin,
                          double pout) {
    EdgeZone z;
    z.hc = z.vc = pout;
    z.hrad = z.hid = z.vrad = z.vis = 0.;
    const double u2 = norm2(u0);
    if (!(u2 > S.rref2 * (1. + 1e-9))) return z;
    const double dir = pout > pin ? 1. : -1., span = fabs(pout - pin), lam = 1.05 * sqrt(u2);
    // Newton's method for f = 0 (stage 0, t = 0: the hidden side), then for the
    // lowest potential on the line = 0 (stage 1, with t: the visible side). A
    // chord of length acc or less answers "not hidden" untested: start inside.
    double w = -0.02 * span, t = 0., vis0 = 0.;
    int stage = 0;
#pragma unroll 1
    for (int it = 0; it < 12; it++) {
        const EdgeEval v = eval_edge(S, u0, u2, acc, pout + dir * w, t);
        const double fp = dir * v.fp;
        if (!v.on || !(fp > 0.) || (stage && !(v.h > 0.))) return z;
        const double dt = stage ? -v.g / v.h : 0.;
        const double m = stage ? v.f + 0.5 * v.g * dt : v.f;  // to second order
        const double s0 = m / fp;
        const double fine = stage ? 5e-4 : 0.05;
        // near enough for the bounds to hold (off below is K s0^2 / fl at least)
        if (s0 * s0 * (kTwoPi * kTwoPi * 2.75) * lam * lam * v.ae <= fine * delta * fp) {
            const EdgeBound B = edge_bound(S, v, lam);
            const double r = sqrt(v.r2);
            double rad = B.rad, K = B.K, fl = fp, extra = 4. * v.tol;
            double gp = 0., move = 0., t3 = 0., cap = 0.;
            bool ok = true;
            if (stage) {
                // curvature along the line keeps 0.6 h while the point moves by
                // at most move (third derivatives of -m / r: 6 m / r^4); the
                // minimum shifts by at most gp rad / hl, gp bounding dg/dphase:
                // the eclipser's part of g is ae t for every phase
                t3 = 9. * (v.ae / r + S.mo * v.io * v.io * v.io * v.io);
                move = 0.4 * v.h / t3;
                if (move > 0.09 * r) move = 0.09 * r;
                if (move * v.io > 0.09) move = 0.09 / v.io;
                const double hl = 0.6 * v.h, tm = fabs(t) + move;
                gp = kTwoPi * (4.2 * v.ae * tm / r * lam + 1.3 * (B.t2 * lam + B.t1));
                K += gp * gp / hl;
                const double rm = (move - fabs(dt)) / (1.2 * kTwoPi * lam + gp / hl);
                if (rm < rad) rad = rm;
                fl -= gp * fabs(v.g) / hl;
                extra += v.g * v.g * (0.5 / hl - 0.5 / v.h);
                ok = tm < 0.5 * lam && dt * dt < 0.25 * (S.rref2 - v.b2);
            } else {
                // inwards the chord only grows: d(b^2)/dw > 0 within rad
                const double db2 = -2. * v.x * v.xp * dir;
                const double rb = 0.5 * db2 / (kTwoPi * kTwoPi * (1.3 * v.b2 + u2));
                if (rb < rad) rad = rb;
                // outwards it shrinks, and one of length acc or less is not searched:
                // d(b^2)/dw w + 2 (2 pi)^2 |u0|^2 w^2 must leave that much
                const double two2u = kTwoPi * kTwoPi * u2;
                const double room =
                    S.rref2 - v.b2 - 0.25 * acc * acc * (1. + 1e-5) - 1e-12 * (1. + u2);
                cap = room / (1.1 * db2);
                if (cap > 0.05 * db2 / two2u) cap = 0.05 * db2 / two2u;
            }
            if (rad * K > 0.8 * fl) rad = 0.8 * fl / K;
            // f (or the minimum) within the zone is f0 + fl w up to K w^2 / 2 and
            // grows with w; past eta from the Newton root it has its sign
            const double eta = (K * s0 * s0 + 2. * extra) / fl;
            const double off = stage ? fabs(s0) * (fp / fl - 1.) + eta : eta;
            if (ok && fl > 0.5 * fp && rad > 0. && K * (fabs(s0) + off) <= 0.2 * fl &&
                fabs(s0) + off < rad && off <= fine * delta) {
                // 4e-15: the rounding of phases near 1
                if (stage) {
                    const double clear = clear_radius(S, u0, v, dir, t, lam, dt, gp / (0.6 * v.h),
                                                      move, off - s0, rad);
                    if (!(fabs(s0) + off < clear)) return z;
                    z.vc = pout + dir * w;
                    z.vrad = clear;
                    z.vis = -s0 + off + 4e-15;
                    const EdgeEnd E{t, dt, v.tol, s0, off, fp, fl, K, rad, gp, move, t3, vis0,
                                    r, v.h, v.ae, v.io, v.b2, v.x, v.ex, v.ey};
                    narrow_zone(S, u0, acc, dir, lam, E, B, z);
                    return z;
                }
                z.hc = pout + dir * w;
                z.hrad = rad;
                z.hid = -s0 - off - 4e-15;
                if (z.hid > 0. && z.hid > cap) z.hid = cap > 0. ? cap : 0.;
                vis0 = -s0 + off + 4e-15;
                stage = 1;
                w -= s0;
                if (v.h > 0.) t = -v.g / v.h;
                if (!(v.h > 0. && 25. * t * t < v.b2)) return z;
                continue;
            }
        }
        w -= s0;
        t += dt;
        if (!(w < 0. && w > -span)) return z;
    }
    return z;
}

// The zones as phases: hidden on [h0, h1], not hidden on [v0, v1] (h0 > h1, v0 > v1:
// nothing), each drawn in by the rounding of its ends.
struct EdgeSpan {
    double h0, h1, v0, v1;
};

LCG_HD EdgeSpan edge_span(const EdgeZone &z, double dir) {
    constexpr double kRound = 2e-15;
    const double ha = z.hc - dir * z.hrad, hb = z.hc + dir * z.hid;
    const double va = z.vc + dir * z.vis, vb = z.vc + dir * z.vrad;
    EdgeSpan e;
    e.h0 = (dir > 0. ? ha : hb) + kRound;
    e.h1 = (dir > 0. ? hb : ha) - kRound;
    e.v0 = (dir > 0. ? va : vb) + kRound;
    e.v1 = (dir > 0. ? vb : va) - kRound;
    if (!(z.hrad > 0.)) { e.h0 = 10.; e.h1 = -10.; }
    if (!(z.vrad > 0.)) { e.v0 = 10.; e.v1 = -10.; }
    return e;
}

LCG_HD int span_test(const EdgeSpan &e, double phase) {
    if (phase >= e.h0 && phase <= e.h1) return kEdgeTrue;
    if (phase >= e.v0 && phase <= e.v1) return kEdgeFalse;
    return kEdgeUnsure;
}

// A phase beyond both intervals' inner ends: only the search tells.
LCG_HD bool span_between(const EdgeSpan &e, double phase) {
    return (phase > e.h1 && phase < e.v0 && e.h0 <= e.h1 && e.v0 <= e.v1) ||
           (phase > e.v1 && phase < e.h0 && e.h0 <= e.h1 && e.v0 <= e.v1);
}

// What the zones say of a phase.
LCG_HD int zone_test(const EdgeZone &z, double dir, double phase) {
    return span_test(edge_span(z, dir), phase);
}

LCG_HD bool zone_between(const EdgeZone &z, double dir, double phase) {
    return span_between(edge_span(z, dir), phase);
}

// ---- the surface radius along a ray ------------------------------------------------

// face_chop (roche.cuh) halves and bisects the radius at which the potential
// along a ray reaches pref: about 27 evaluations of a square root and two
// divisions. Along the ray the potential is, about the star's centre,
//   f(r) = -me / r - mo / d - ss/2 (dx^2 + dy^2) r^2 + k dx r - pref,
//   d^2 = r^2 + 1 - 2 S.dx dx r,
// and concave while 2 me / r^3 > mo / (1 - r)^3 (checked at rref, where the left
// side is least). With f'(rref) > 0 it then increases on (0, rref], so its root
// decides every comparison of face_chop: Newton's method from rref lands left
// of the root once and climbs (a concave function lies under its tangents), and
// a value e <= 0 at r encloses it in [r - e / f'(r), r - e / f'(rref)], f' being
// between the two from there on. The radius is face_chop's, bit for bit: the
// same midpoints, those inside the enclosure (1e-13 wide, far below acc) by
// chop_pot itself. 4-5 evaluations replace 27; where a condition fails (the
// ray through L1 of a lobe-filling star), face_chop runs as it is.
LCG_HD int face_chop_root(const EdgeStar &S, int star, double q, double spin, double dx, double dy,
                          double rref, double pref, double acc, double &rad) {
    const double dxy2 = dx * dx + dy * dy, sd = S.dx * dx, kd = S.k * dx;
    double tol = 0.;
    auto eval = [&](double r, double &f, double &d1) {
        const double ir = 1. / r, io = edge_rsqrt(fma(r, r - 2. * sd, 1.));
        const double pe = S.me * ir, po = S.mo * io;
        f = fma(kd, r, fma(-0.5 * S.ss * dxy2, r * r, -(pe + po))) - S.pref;
        d1 = fma(pe, ir, fma(po * io * io, r - sd, fma(-S.ss * dxy2, r, kd)));
        tol = 1e-14 * (pe + po + 2.);
    };
    const double gap = 1. - rref;
    double f, d1;
    eval(rref, f, d1);
    const double dmin = d1;
    bool ok = gap > 0.1 && 2. * S.me * gap * gap * gap > S.mo * rref * rref * rref && dmin > 0. &&
              f > 4. * tol;
    double lo = 0., hi = 0.;
    if (ok) {
        double r = rref;
        ok = false;
#pragma unroll 1
        for (int it = 0; it < 12; it++) {
            r -= f / d1;
            if (!(r > 0.)) break;
            eval(r, f, d1);
            if (!(d1 > 0.)) break;
            if (f <= tol && (tol - f) < 1e-2 * acc * dmin) {
                // f is at most 0 up to rounding: both ends with 2 tol to spare
                const double e = f < 0. ? -f : 0.;
                lo = r + (e - 2. * tol) / d1 - 2. * tol / dmin;
                hi = r + (e + 4. * tol) / dmin;
                ok = true;
                break;
            }
        }
    }
    if (!ok) return face_chop(star, q, spin, dx, dy, rref, pref, acc, rad);
    // face_chop's walk; pot(r) < pref left of lo, > pref right of hi
    double r1 = rref / 2, r2 = rref;
    bool above = true;
    for (int it = 0; it < 30 && above; it++) {
        r1 = r2 / 2;
        above = r1 < lo ? false : r1 > hi ? true : chop_pot(star, q, spin, dx, dy, r1) > pref;
        if (above) r2 = r1;
    }
    int fail = above ? 2 : 0;
    if (!fail) {
        for (int nchop = 0; nchop < 100 && r2 - r1 > acc; nchop++) {
            const double r = (r1 + r2) / 2.;
            const bool below =
                r < lo ? true : r > hi ? false : chop_pot(star, q, spin, dx, dy, r) < pref;
            if (below) r1 = r;
            else r2 = r;
        }
        if (r2 - r1 > acc) fail = 3;
    }
    rad = (r1 + r2) / 2.;
    return fail;
}

}  // namespace lcg
