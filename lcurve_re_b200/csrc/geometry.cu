// geometry.cu — the FP64 stages of one light curve, compiled with
// --fmad=false so that every product and sum rounds as in the reference:
//   k_grid       face radius solve, normal, gravity, area (set_star_grid.cpp:226-523)
//   k_ecl_*      sphere pre-test, Roche eclipse candidates, their ingress and egress
//   k_continuum  gravity darkening, irradiation, black body (set_star_continuum.cpp),
//                sums behind logg and the volume-averaged radius (comp_gravity.cpp,
//                comp_radius.cpp)
//   k_flat_*     stable partition into FlatGrid order (comp_light_flat.cpp:26-65)
//   k_phases     per-point phase and sub-exposure entries (light_curve_comp.cpp:350-455)
//   k_scatter    merge of the flux partials into the light curve (:457-498)
//   k_run_bounds* the sweeps' records of face groups
//   k_finalize   scale factor and chi**2 (re_scale.cpp:16-42, light_curve_comp.cpp:557-585)
#include <stdlib.h>

#include "eclipse.cuh"
#include "engine.h"
#include "fixed_phase.cuh"

namespace lcg {

namespace {

__device__ __forceinline__ void set_status(DevStatus *st, int code, int64_t face) {
    if (atomicCAS(&st->code, 0, code) == 0) st->face = (int32_t)face;
}

// The largest k < n with at(k) <= u, at(0) <= u, for a whole warp at once: 32 entries
// a step, so two dependent loads for a thousand entries instead of a binary
// search's ten. The faces of 256 models of 60-400 strips: 1.21 -> 1.05 ms, their
// sphere tests 0.36 -> 0.32; the queued candidates of the eclipse stage, whose lanes
// do not follow one another, lose 2% by it and keep find_seg.
template <class At>
__device__ __forceinline__ int warp_search(int n, int64_t u, const At &at) {
    const int lane = threadIdx.x & 31;
    int lo = 0;
    while (n > 1) {
        const int step = (n + 31) >> 5, o = lane * step;
        const unsigned m = __ballot_sync(0xffffffffu, o < n && at(lo + o) <= u);
        const int j = (31 - __clz(m)) * step;
        lo += j;
        n = n - j < step ? n - j : step;
    }
    return lo;
}

// One half-face h of a grid and its mirror partner; lo: its ring or an earlier one.
__device__ __forceinline__ void grid_half(const GridParams &p, const RingRec *__restrict__ rings,
                                          GridDev g, int64_t h, int lo, DevStatus *st) {
    while (lo + 1 < p.nrings && rings[lo + 1].hoff <= h) lo++;
    const RingRec R = rings[lo];
    const int np = (int)(h - R.hoff);
    const double phi = R.phi1 + R.span * (np + 0.5) / R.nphi;
    const double sinp = sin(phi), cosp = cos(phi);
    const V3 dirn = p.npole ? v3(R.sint * cosp, R.sint * sinp, R.cost)
                            : v3(R.cost, R.sint * cosp, R.sint * sinp);
    const V3 cofm = p.star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
    double rad, gravity;
    V3 posn, dvec;
    if (p.roche) {
        const int fail = face_chop_root(p.own, p.star, p.q, p.spin, dirn.x, dirn.y, p.rref, p.pref,
                                        p.acc, rad);
        if (fail) {
            // the reference re-runs the scalar Roche::face on such lanes
            if (face_scalar(p.star, p.q, p.spin, dirn, p.rref, p.pref, p.acc, posn, dvec, rad,
                            gravity)) {
                set_status(st, 3, R.off + np);
                return;
            }
        } else {
            posn = add(cofm, scale(rad, dirn));
            dvec = drpot(p.star, p.q, p.spin, posn);
            gravity = len(dvec);
            dvec.x /= gravity;
            dvec.y /= gravity;
            dvec.z /= gravity;
        }
    } else {
        rad = p.rad_sphere;
        posn = add(cofm, scale(rad, dirn));
        dvec = dirn;
        gravity = 1.;
    }
    const double area = (R.span / R.nphi * rad * R.sint) * (R.latspan / R.nl * rad) / dot(dirn, dvec);
    const float af = (float)area, gf = (float)(gravity / p.gref);
    // a tiled face past the reference's face count is dropped (its vector
    // ends there, set_star_grid.cpp:162-166)
    int64_t i = R.off + np;
    if (i < g.n) {
        g.px[i] = posn.x; g.py[i] = posn.y; g.pz[i] = posn.z;
        g.nx[i] = dvec.x; g.ny[i] = dvec.y; g.nz[i] = dvec.z;
        g.area[i] = af;
        g.grav[i] = gf;
    }
    const int np2 = R.nphi - 1 - np;
    if (np2 != np && R.off + np2 < g.n) {
        i = R.off + np2;
        if (p.npole) {
            g.px[i] = posn.x; g.py[i] = -posn.y; g.pz[i] = posn.z;
            g.nx[i] = dvec.x; g.ny[i] = -dvec.y; g.nz[i] = dvec.z;
        } else {
            g.px[i] = posn.x; g.py[i] = posn.y; g.pz[i] = -posn.z;
            g.nx[i] = dvec.x; g.ny[i] = dvec.y; g.nz[i] = -dvec.z;
        }
        g.area[i] = af;
        g.grav[i] = gf;
    }
}

// Also clears the eclipse stage's eight work counters.
__global__ void k_grid(GridParams p, const RingRec *__restrict__ rings, GridDev g,
                       int32_t *counters, DevStatus *st) {
    const int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (h < 8) counters[h] = 0;
    const int64_t h0 = h & ~31ll;
    if (h0 >= p.nhalf) return;  // whole warps
    const int lo = warp_search(p.nrings, h0, [&](int i) { return (int64_t)rings[i].hoff; });
    if (h < p.nhalf) grid_half(p, rings, g, h, lo, st);
}

// Sphere test of face i: a spherical eclipser sets the range directly; a
// Roche eclipser makes the face a candidate. kZero: the range of a face that is
// never eclipsed is written as zeros (grids that callers read).
template <bool kZero>
__device__ __forceinline__ bool ecl_pre_face(const EclParams &p, int32_t eclipse_on, GridDev g,
                                             int64_t i) {
    bool cand = false;
    if (i >= g.ntiled) {
        // a default Point (lcurve.h:53-54): no face of the tiling lands here
        g.px[i] = g.py[i] = g.pz[i] = 0.;
        g.nx[i] = g.ny[i] = g.nz[i] = 0.;
        g.area[i] = 0.f;
        g.grav[i] = 1.f;
        g.necl[i] = 0;
        g.ein[i] = g.eout[i] = 0.;
    } else {
        g.necl[i] = 0;
        if constexpr (kZero) {
            g.ein[i] = 0.;
            g.eout[i] = 0.;
        }
        if (eclipse_on) {
            const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
            const V3 cofm = p.comp_star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
            double phi1, phi2, lam1, lam2;
            if (p.comp_roche) {
                cand = sphere_eclipse_ph(p.cosi, p.sini, pos, cofm, p.comp_rref, phi1, phi2,
                                         lam1, lam2);
            } else if (sphere_eclipse_ph(p.cosi, p.sini, pos, cofm, p.comp_r, phi1, phi2, lam1,
                                         lam2)) {
                g.necl[i] = 1;
                g.ein[i] = phi1;
                g.eout[i] = phi2;
            }
        }
    }
    return cand;
}

// Appends the candidates of a full warp to the queue (warp-aggregated).
__device__ __forceinline__ void queue_push(bool cand, int32_t item, int32_t *queue,
                                           int32_t *counters) {
    const unsigned mask = __ballot_sync(0xffffffffu, cand);
    if (mask) {
        const int lane = threadIdx.x & 31;
        const int leader = __ffs(mask) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(&counters[0], __popc(mask));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (cand) queue[base + __popc(mask & ((1u << lane) - 1u))] = item;
    }
}

// Sphere test of every face; Roche eclipsers queue their candidates.
__global__ void k_ecl_pre(EclParams p, int32_t eclipse_on, GridDev g, int32_t *queue,
                          int32_t *counters) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool cand = i < g.n && ecl_pre_face<true>(p, eclipse_on, g, i);
    queue_push(cand, (int32_t)i, queue, counters);
}

// Ingress/egress of the queued candidates, one warp per face
// (ingress_egress_warp), for calls that ask for it with at most warp_max
// candidates: the plain bisection, which the tests compare the thread mode
// with. Otherwise k_ecl_potmin and k_ecl_bisect do the work (one thread per
// candidate, each warp taking 32 consecutive candidates at a time so that
// neighbouring faces, with similar iteration counts, run in lockstep) and this
// kernel is not launched, or returns at once: the count is read on the device.
__global__ void __launch_bounds__(128, 4) k_ecl_roche(EclParams p, GridDev g,
                                                   const int32_t *__restrict__ queue,
                                                   int32_t *counters, DevStatus *st,
                                                   int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = counters[0];
    if (total <= warp_max) {
        for (;;) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&counters[1], 1);
            k = __shfl_sync(full, k, 0);
            if (k >= total) break;
            const int32_t i = queue[k];
            const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
            double ing = 0., egr = 0.;
            int s = 0;
            const bool ecl = ingress_egress_warp(p.comp_star, p.q, p.comp_spin, p.cosi, p.sini,
                                                 p.delta, pos, p.comp_rref, p.comp_pref, ing,
                                                 egr, s);
            if (lane == 0) {
                if (s) {
                    set_status(st, s, i);
                } else if (ecl) {
                    g.necl[i] = 1;
                    g.ein[i] = ing;
                    g.eout[i] = egr;
                }
            }
        }
        return;
    }
}

// Appends the eclipsed candidates k of a warp's 32 (lanes with hit) to the
// list the bisection pass walks, in lane order, so that warps bisect only
// faces pot_min found eclipsed (consecutive candidates stay together). All 32
// lanes call it.
__device__ __forceinline__ void push_hits(bool hit, int k, int32_t *hits, int32_t *count) {
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (lane == 0) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (hit) hits[at + __popc(m & ((1u << lane) - 1u))] = k;
}

// Thread mode (more candidates than warp_max), in two passes with a small code
// footprint each, as for the batch (k_ecl_potmin_b / k_ecl_bisect_b): the
// sphere test and pot_min per candidate, then ingress and egress on the two
// lanes of a pair. es holds each candidate's state between the passes, hits
// the candidates pot_min found eclipsed.
__global__ void __launch_bounds__(128, 4) k_ecl_potmin(EclParams p, GridDev g,
                                                    const int32_t *__restrict__ queue,
                                                    int32_t *counters, double4 *es, int32_t *hits,
                                                    DevStatus *st, int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = counters[0];
    if (total <= warp_max) return;
    const V3 cofm = p.comp_star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&counters[2], 32);
        base = __shfl_sync(full, base, 0);
        if (base >= total) break;
        const int k = base + lane;
        bool hit = false;
        if (k < total) {
            const int32_t i = queue[k];
            const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
            double phi1, phi2, lam1, lam2, phi = 0., lam = 0.;
            if (sphere_eclipse_ph(p.cosi, p.sini, pos, cofm, p.comp_rref, phi1, phi2, lam1,
                                  lam2)) {
                const double ACC = 2. * sqrt(2. * kTwoPi * (lam2 - lam1) * p.delta);
                int s = 0;
                hit = pot_min(p.comp_star, p.q, p.comp_spin, p.cosi, p.sini, pos, phi1, phi2,
                              lam1, lam2, p.comp_rref, p.comp_pref, ACC, phi, lam, s);
                if (s) {
                    set_status(st, s, i);
                    hit = false;
                }
                es[k] = make_double4(phi, phi1, phi2, ACC);
            }
        }
        push_hits(hit, k, hits, &counters[6]);
    }
}

template <int NB>
__global__ void __launch_bounds__(128, NB)
    k_ecl_bisect(__grid_constant__ const EclParams p, __grid_constant__ const GridDev g,
                 const int32_t *__restrict__ queue, int32_t *counters, const double4 *es,
                 const int32_t *__restrict__ hits, DevStatus *st, int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = counters[0];
    if (total <= warp_max) return;
    const int64_t n2 = 2 * (int64_t)counters[6];
    for (;;) {
        int64_t base = 0;
        if (lane == 0) base = atomicAdd(&counters[3], 32);
        base = __shfl_sync(full, base, 0);
        if (base >= n2) break;
        // every lane stays here (bisect_warp votes over the warp); both
        // lanes of a pair agree on live
        const int64_t u = base + lane;
        const int side = (int)(u & 1);
        const bool live = u < n2;
        const int k = live ? hits[u >> 1] : 0;
        const int32_t i = live ? queue[k] : 0;
        const double4 E = live ? es[k] : make_double4(0., 0., 0., 0.);
        const V3 pos = live ? v3(g.px[i], g.py[i], g.pz[i]) : v3(0., 0., 0.);
        int s = 0;
        double v = bisect_warp(p, live, E.x, side ? E.z : E.y, E.w, pos, s);
        v = v - floor(v);
        const double other = __shfl_xor_sync(full, v, 1);
        const int os = __shfl_xor_sync(full, s, 1);
        if (live && side == 0) {
            if (s || os) {
                set_status(st, s ? s : os, i);
            } else {
                double egr = other;
                if (egr < v) egr++;
                g.necl[i] = 1;
                g.ein[i] = v;
                g.eout[i] = egr;
            }
        }
    }
}

// The whole eclipse stage of a grid small enough that two lanes per face fit the
// GPU at once: sphere test, pot_min (both lanes of a pair, in step) and the
// boundaries, one lane each. The three kernels and the candidate queue of larger
// grids keep warps full, which nothing is gained by here: 8,152 faces 36 us in
// three launches -> 24 in one.
__global__ void __launch_bounds__(128, 4)
    k_ecl_small(__grid_constant__ const EclParams p, int32_t eclipse_on,
                __grid_constant__ const GridDev g, DevStatus *st) {
    const unsigned full = 0xffffffffu;
    const int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t i = u >> 1;
    const int side = (int)(u & 1);
    // lane 0 of a pair writes the face's defaults and says whether it is a candidate
    bool cand = side == 0 && i < g.n && ecl_pre_face<true>(p, eclipse_on, g, i);
    cand = __shfl_sync(full, cand, threadIdx.x & 30);
    if (!__any_sync(full, cand)) return;
    const V3 cofm = p.comp_star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
    const V3 pos = cand ? v3(g.px[i], g.py[i], g.pz[i]) : v3(0., 0., 0.);
    double phi1 = 0., phi2 = 0., lam1 = 0., lam2 = 0., phi = 0., lam = 0., acc = 0.;
    bool live = false;
    int s = 0;
    if (cand &&
        sphere_eclipse_ph(p.cosi, p.sini, pos, cofm, p.comp_rref, phi1, phi2, lam1, lam2)) {
        acc = 2. * sqrt(2. * kTwoPi * (lam2 - lam1) * p.delta);
        live = pot_min(p.comp_star, p.q, p.comp_spin, p.cosi, p.sini, pos, phi1, phi2, lam1, lam2,
                       p.comp_rref, p.comp_pref, acc, phi, lam, s);
        if (s) live = false;
    }
    double v = bisect_warp(p, live, phi, side ? phi2 : phi1, acc, pos, s);
    v = v - floor(v);
    const double other = __shfl_xor_sync(full, v, 1);
    const int os = __shfl_xor_sync(full, s, 1);
    if (!cand || side) return;
    if (s || os) {
        set_status(st, s ? s : os, i);
    } else if (live) {
        double egr = other;
        if (egr < v) egr++;
        g.necl[i] = 1;
        g.ein[i] = v;
        g.eout[i] = egr;
    }
}

// The flux of face i (set_star_continuum.cpp:26-297).
__device__ __forceinline__ float continuum_flux(const ContParams &p, const GridDev &g, int64_t i) {
    if (i >= g.ntiled) return 0.f;  // default Point: zero area, zero flux
    const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
    const V3 dir = v3(g.nx[i], g.ny[i], g.nz[i]);
    const V3 cofm_other = p.star == kStar1 ? v3(1., 0., 0.) : v3(0., 0., 0.);
    const V3 vec = sub(cofm_other, pos);
    const double r = len(vec);
    const double mu = dot(dir, vec) / r;
    const double EFAC = p.efac;
    double t;
    if (p.star == kStar1) {
        t = p.t_own;
        for (int k = 0; k < p.nspot; k++) {
            const V3 sd = v3(p.spot_dir[k][0], p.spot_dir[k][1], p.spot_dir[k][2]);
            double dist = rad2deg(acos(dot(pos, sd) / len(pos)));
            t += (p.spot_tcen[k] - p.t_own) * exp(-sq(dist / (p.spot_fwhm[k] / EFAC)) / 2.);
        }
        if (p.uesp_on) {
            const V3 evec = v3(pos.x, pos.y, 0);
            const double evecl = len(evec);
            if (evecl > 0.) {
                double rd = len(pos);
                double clat = dot(pos, evec) / evecl / rd;
                clat = dmin(1.0, dmax(-1., clat));
                double dlat = rad2deg(acos(clat));
                double clong = dot(v3(p.uesp_dir[0], p.uesp_dir[1], p.uesp_dir[2]), evec) / evecl;
                clong = dmin(1.0, dmax(-1., clong));
                double dlong = rad2deg(acos(clong));
                if (dlat <= p.uesp_lathw && dlong <= p.uesp_longhw) {
                    t = p.uesp_temp;
                } else if (dlat <= p.uesp_lathw) {
                    t += (p.uesp_temp - p.t_own) * exp(-(dlong - p.uesp_longhw) / p.uesp_taper);
                } else if (dlong <= p.uesp_longhw) {
                    t += (p.uesp_temp - p.t_own) * exp(-(dlat - p.uesp_lathw) / p.uesp_taper);
                } else {
                    t += (p.uesp_temp - p.t_own) * exp(-(dlat - p.uesp_lathw) / p.uesp_taper) *
                         exp(-(dlong - p.uesp_longhw) / p.uesp_taper);
                }
            }
        }
    } else {
        t = fabs(p.t_own);
        for (int k = 0; k < p.nspot; k++) {
            const V3 sd = v3(p.spot_dir[k][0], p.spot_dir[k][1], p.spot_dir[k][2]);
            const V3 off = sub(pos, v3(1., 0., 0.));
            double dist = rad2deg(acos(dot(off, sd) / len(off)));
            t += (p.spot_tcen[k] - t) * exp(-sq(dist / (p.spot_fwhm[k] / EFAC)) / 2.);
        }
    }
    if (p.fp32) {
        // the intensity in FP32 (the face's flux is stored as a float): the same
        // formulas as below; x^(1/4) as two square roots, Planck from its
        // constants over the wavelength, set on the host
        const float gd = powf(g.grav[i], (float)p.gdcbol);
        const float tg = (float)t * gd, tg2 = tg * tg;
        const double rc = p.rcomp;
        double geom = 0.;
        float temp = tg;
        if (mu > -rc) {
            if (mu >= rc) {
                geom = sq(rc / r) * mu;
            } else {
                double x0 = -mu / rc;
                geom = sq(rc / r) * rc *
                       (sqrt(1. - x0 * x0) * (2 + x0 * x0) / 3 - x0 * (kPi / 2 - asin(x0))) / kPi;
            }
            temp = sqrtf(sqrtf(fmaf(tg2, tg2, p.irr32 * (float)geom)));
        }
        const float area = g.area[i];
        float f = area * (p.planck_c1 / (expf(p.planck_c2 / temp) - 1.f));
        if (p.mirror) {
            const float tm = (float)(p.star == kStar1 ? fabs(p.t_other) : p.t_other);
            f = fmaf(area * (float)geom, p.planck_c1 / (expf(p.planck_c2 / tm) - 1.f), f);
        }
        return f;
    }
    const double gd = pow((double)g.grav[i], p.gdcbol);
    const double rc = p.rcomp;
    // pow(t_other, 4) for star 1 and pow(t_other, 4.) for star 2 are the same call
    const double irr = p.absorb * pow(p.t_other, 4.);
    double temp, geom;
    if (mu >= rc) {
        geom = sq(rc / r) * mu;
        temp = pow(pow(t * gd, 4.0) + irr * geom, 0.25);
    } else if (mu > -rc) {
        double x0 = -mu / rc;
        geom = sq(rc / r) * rc * (sqrt(1. - x0 * x0) * (2 + x0 * x0) / 3 - x0 * (kPi / 2 - asin(x0))) /
               kPi;
        temp = pow(pow(t * gd, 4.0) + irr * geom, 0.25);
    } else {
        geom = 0.;
        temp = t * gd;
    }
    float f = (float)(g.area[i] * planck(p.wavelength, temp));
    if (p.mirror) {
        const double tm = p.star == kStar1 ? fabs(p.t_other) : p.t_other;
        f = (float)(f + g.area[i] * geom * planck(p.wavelength, tm));
    }
    return f;
}

constexpr int kContBlock = 256;  // faces per CTA of k_continuum and of the partition counts
constexpr int kFlatBlock = 1024;

// Eclipse class of face i for the FlatGrid partition (comp_light_flat.cpp:26-65):
// 0 never eclipsed, 1 one range, 2 several (an opaque disc's ranges added to
// the companion's).
__device__ __forceinline__ int flat_class(const GridDev &g, int64_t i) {
    const int k = g.necl[i] + (g.ndx ? g.ndx[i] : 0);
    return k < 2 ? k : 2;
}

// Face fluxes, and while the face is in registers what later stages would read
// it again for: per CTA of 256 faces the number of one-range faces (cnt, for
// k_flat_scatter; an opaque disc's ranges replace the counts, k_disc_faces) and
// the sums behind log g and the volume-averaged radius (comp_gravity.cpp:20-155,
// comp_radius.cpp:16-86: f g, f, solid angle, volume) as four doubles (dsum), a
// fixed tree. Either may be null. A pass of its own over the faces took 8 us on
// 10,300 faces and 25 us on 865,000; here they add 0.6 and 7.
__global__ void __launch_bounds__(kContBlock) k_continuum(ContParams p, GridDev g, int32_t *cnt,
                                                          double *dsum) {
    const int64_t i = blockIdx.x * (int64_t)kContBlock + threadIdx.x;
    const bool in = i < g.n;
    double v[4] = {0., 0., 0., 0.};
    if (in) {
        const float f = continuum_flux(p, g, i);
        g.flux[i] = f;
        v[0] = (double)(f * g.grav[i]);
        v[1] = (double)f;
        const V3 vec = v3(g.px[i] - (p.star == kStar1 ? 0. : 1.), g.py[i], g.pz[i]);
        const double r = len(vec);
        v[3] = g.area[i] * dot(v3(g.nx[i], g.ny[i], g.nz[i]), vec);
        v[2] = v[3] / (r * r * r);
    }
    if (cnt) {
        const int c = __syncthreads_count(in && g.necl[i] == 1);
        if (threadIdx.x == 0) {
            cnt[blockIdx.x] = c;
            cnt[gridDim.x + blockIdx.x] = 0;
        }
    }
    if (!dsum) return;
    __shared__ double sh[kContBlock / 32][4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        if (lane == 0) sh[w][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0.;
        for (int k = 0; k < kContBlock / 32; k++) s += sh[k][threadIdx.x];
        dsum[4 * (int64_t)blockIdx.x + threadIdx.x] = s;
    }
}

// Single block: exclusive scan of the per-block eclipse counts; n0 = faces
// never eclipsed.
__device__ __forceinline__ void scan_blocks(int32_t *blockcnt, int32_t nb, int64_t n,
                                            int64_t *n0) {
    __shared__ int32_t part[1024];
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? blockcnt[i] : 0;
        part[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            int t = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
            __syncthreads();
            part[threadIdx.x] += t;
            __syncthreads();
        }
        if (i < nb) blockcnt[i] = (int32_t)(carry + part[threadIdx.x] - v);
        __syncthreads();
        if (threadIdx.x == 1023) carry += part[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) *n0 = n - carry;
    __syncthreads();
}

// Face i's record of the fast mixed sweep at flat position dest (pairs of
// faces interleaved, FlatDev::fp).
__device__ __forceinline__ void fast_record(float *fp, int64_t dest, GridDev g, int64_t i,
                                            const FastCoef &fc) {
    const double fl = (double)g.flux[i];
    float *r = fp + 16 * (dest >> 1) + (dest & 1);
    r[0] = (float)g.nx[i];
    r[2] = (float)g.ny[i];
    r[4] = (float)(fc.cosi * g.nz[i]);
    r[6] = (float)(fl * fc.p[0]);
    r[8] = (float)(fl * fc.p[1]);
    r[10] = (float)(fl * fc.p[2]);
    r[12] = (float)(fl * fc.p[3]);
    r[14] = (float)(fl * fc.p[4]);
}

// Stable three-way partition [never | one range | several]. Several-range
// faces get all-zero records (they add exact zeros to the main sweeps) and
// their face index and ranges in FlatGrid order; k_flux_ragged adds them. Each
// CTA adds up the counts before its block itself (at most a few thousand, 16 KB
// from L2), which spares the two launches that counted and scanned; CTA 0
// stores n0 and n1. CTAs past the last face zero the fast records up to npad.
__global__ void __launch_bounds__(kFlatBlock) k_flat_scatter(GridDev g, FlatDev f,
                                                             const int32_t *__restrict__ cnt,
                                                             int32_t ncnt, int mixed, int need_pos,
                                                             FastCoef fc) {
    __shared__ int32_t warp_tot[2][32], red[32][4];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int64_t i = blockIdx.x * (int64_t)kFlatBlock + t;
    const bool in = i < g.n;
    // one- and several-range faces before this block, and of the grid
    const int mine = (int)blockIdx.x * (kFlatBlock / kContBlock);
    int sum[4] = {0, 0, 0, 0};
    for (int k = t; k < ncnt; k += kFlatBlock) {
        const int c1 = cnt[k], c2 = cnt[ncnt + k];
        sum[2] += c1;
        sum[3] += c2;
        if (k < mine) {
            sum[0] += c1;
            sum[1] += c2;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        for (int o = 16; o > 0; o >>= 1) sum[q] += __shfl_down_sync(0xffffffffu, sum[q], o);
        if (lane == 0) red[w][q] = sum[q];
    }
    const int cls = in ? flat_class(g, i) : 0;
    const unsigned m1 = __ballot_sync(0xffffffffu, cls == 1);
    const unsigned m2 = __ballot_sync(0xffffffffu, cls == 2);
    if (lane == 0) {
        warp_tot[0][w] = __popc(m1);
        warp_tot[1][w] = __popc(m2);
    }
    __syncthreads();
    // every warp adds the 32 partial sums the same way
#pragma unroll
    for (int q = 0; q < 4; q++) {
        int v = red[lane][q];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        sum[q] = v;
    }
    const int64_t boff1 = sum[0], boff2 = sum[1];
    const int64_t n1 = g.n - sum[3], n0 = n1 - sum[2];
    if (blockIdx.x == 0 && t == 0) {
        f.n0[0] = n0;
        f.n0[1] = n1;
    }
    int b1 = 0, b2 = 0;
    for (int k = 0; k < w; k++) {
        b1 += warp_tot[0][k];
        b2 += warp_tot[1][k];
    }
    const unsigned below = (1u << lane) - 1u;
    const int rank1 = b1 + __popc(m1 & below), rank2 = b2 + __popc(m2 & below);
    if (!in) {
        if (mixed && fc.on && i < f.npad) {  // padding adds nothing
            float *r = f.fp + 16 * (i >> 1) + (i & 1);
            for (int q = 0; q < 16; q += 2) r[q] = 0.f;
        }
        return;
    }
    const int64_t dest = cls == 1   ? n0 + boff1 + rank1
                         : cls == 2 ? n1 + boff2 + rank2
                                    : blockIdx.x * (int64_t)kFlatBlock - boff1 - boff2 +
                                          (t - rank1 - rank2);
    // a one-range face's range: the companion's, else the disc's first
    double ein = 0., eout = 0.;
    if (cls == 1) {
        if (g.necl[i]) { ein = g.ein[i]; eout = g.eout[i]; }
        else { ein = g.xr[kDiscRanges * i].x; eout = g.xr[kDiscRanges * i].y; }
    }
    const bool live = cls < 2;
    if (mixed) {
        if (fc.on) {
            if (live) {
                fast_record(f.fp, dest, g, i, fc);
            } else {
                float *r = f.fp + 16 * (dest >> 1) + (dest & 1);
                for (int q = 0; q < 16; q += 2) r[q] = 0.f;
            }
        } else {
            f.geo[dest] = live ? make_float4((float)g.nx[i], (float)g.ny[i], (float)g.nz[i],
                                             g.flux[i])
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        f.ecl[dest] = cls == 1 ? ecl_fx64(ein, eout) : make_ulonglong2(0ull, 0ull);
        if (need_pos)
            f.pos[dest] = live ? make_float4((float)g.px[i], (float)g.py[i], (float)g.pz[i], 0.f)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        const double z = 0.;
        f.dx[dest] = live ? g.nx[i] : z; f.dy[dest] = live ? g.ny[i] : z;
        f.dz[dest] = live ? g.nz[i] : z;
        f.px[dest] = live ? g.px[i] : z; f.py[dest] = live ? g.py[i] : z;
        f.pz[dest] = live ? g.pz[i] : z;
        f.flux[dest] = live ? (double)g.flux[i] : z;
        f.in1[dest] = ein;
        f.out1[dest] = eout;
    }
    if (cls == 2) {
        const int64_t r = dest - n1;
        int q = 0;
        if (g.necl[i]) f.rr[kRagRanges * r + q++] = make_double2(g.ein[i], g.eout[i]);
        for (int k = 0; k < g.ndx[i]; k++) f.rr[kRagRanges * r + q++] = g.xr[kDiscRanges * i + k];
        f.rn[r] = (uint8_t)q;
        f.ridx[r] = (int32_t)i;
    }
}

// Orbital phase of one point (4 Newton steps with pdot, the deltat shift)
// and its polynomial scale factor (light_curve_comp.cpp:358-376).
__device__ __forceinline__ void point_phase(const PhaseParams &p, const DatumRec &d,
                                            double &phase, double &slfac) {
    phase = (d.time - p.t0) / p.period;
    for (int it = 0; it < 4; it++)
        phase -= (p.t0 + phase * (p.period + p.pdot * phase) - d.time) /
                 (p.period + 2. * p.pdot * phase);
    phase += p.deltat / p.period / 2. * (cos(2. * kPi * phase) - 1.);
    const double frac = (d.time - p.middle) / p.range;
    slfac = 1. + frac * (p.slope + frac * (p.quad + frac * p.cube));
}

// Phase and trapezoid weight of sub-exposure nd (light_curve_comp.cpp:416-455).
__device__ __forceinline__ void sub_exposure(double phase, double expose, int ndiv, int nd,
                                             double &phi, double &wgt) {
    if (ndiv == 1) {
        phi = phase;
        wgt = 1.0;
    } else {
        phi = phase + expose * (nd - (ndiv - 1) / 2.0) / (ndiv - 1);
        wgt = (nd == 0 || nd == ndiv - 1) ? 0.5 : 1.0;
    }
}

// The point's sub-exposure entries; with extra, one more entry after the last
// point's (the phase-0.5 entry of wdwarf, light_curve_comp.cpp:504-508: its earth
// vector and phase are given, its weights unused).
__global__ void k_phases(PhaseParams p, const DatumRec *__restrict__ data,
                         const int64_t *__restrict__ off, int32_t n, PhaseDev ph, int32_t extra,
                         V3 ew, double phw) {
    const int np = blockIdx.x * blockDim.x + threadIdx.x;
    if (np == n && extra) {
        const int64_t e = off[n];
        ph.ex[e] = ew.x;
        ph.ey[e] = ew.y;
        ph.ez[e] = ew.z;
        ph.phin[e] = phw;
        ph.ef[e] = make_float4((float)ew.x, (float)ew.y, (float)ew.z, 0.f);
        ph.pfx[e] = phase_fx64(phw);
    }
    if (np >= n) return;
    const DatumRec d = data[np];
    double phase, slfac;
    point_phase(p, d, phase, slfac);
    const double expose = d.expose / p.period;
    const int ndiv = d.ndiv;
    const double norm = (ndiv - 1 > 1) ? ndiv - 1 : 1;
    int64_t e = off[np];
    for (int nd = 0; nd < ndiv; ++nd, ++e) {
        double phi, wgt;
        sub_exposure(phase, expose, ndiv, nd, phi, wgt);
        const V3 earth = set_earth(p.cosi, p.sini, phi);
        const double phin = phi - floor(phi);
        ph.ex[e] = earth.x;
        ph.ey[e] = earth.y;
        ph.ez[e] = earth.z;
        ph.phin[e] = phin;
        ph.w1[e] = slfac * wgt * gi_scale1(p.gi, phi) / norm;
        ph.w2[e] = slfac * wgt * gi_scale2(p.gi, phi) / norm;
        ph.type[e] = (uint8_t)gi_type(p.gi, phi);
        ph.ef[e] = make_float4((float)earth.x, (float)earth.y, (float)earth.z, 0.f);
        ph.pfx[e] = phase_fx64(phin);
    }
}

// v[0] + v[ldp] + ... over nc rows in order, 32 loads in flight: a thread's sum
// is bound by their latency (100 rows: 7.6 us with 8, 4.6 with 32).
__device__ __forceinline__ double sum_rows(const double *__restrict__ v, int64_t nc, int64_t ldp) {
    double o = 0.0;
    int64_t c = 0;
    for (; c + 32 <= nc; c += 32) {
        double x[32];
#pragma unroll
        for (int u = 0; u < 32; u++) x[u] = v[(c + u) * ldp];
#pragma unroll
        for (int u = 0; u < 32; u++) o += x[u];
    }
    for (; c + 4 <= nc; c += 4) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = v[(c + u) * ldp];
#pragma unroll
        for (int u = 0; u < 4; u++) o += x[u];
    }
    for (; c < nc; c++) o += v[c * ldp];
    return o;
}

// Sum of the chunk partials of every phase entry. G = 1: chunks in order (for the
// FP64 sweep: the reference's block order), one thread per (sweep, entry);
// consecutive threads read consecutive entries of a chunk row. G = 8 (mixed
// sweeps): eight warps take eighths of the rows and their sums are added in
// order, eight times the loads in flight: 796 rows of 25,000 entries 72 -> 38 us,
// 130 rows of 500 7.4 -> 2.8.
template <int G>
__global__ void __launch_bounds__(256) k_reduce_chunks(ReduceParams p) {
    constexpr int W = 256 / G;  // entries per CTA
    const int s = blockIdx.y;
    const int x = threadIdx.x % W, y = threadIdx.x / W;
    const int64_t e = blockIdx.x * (int64_t)W + x;
    const double *__restrict__ part = p.part[s];
    if (!part) return;
    const bool in = e < p.nent[s];
    const int64_t nc = p.nchunk[s], ldp = p.ldp;
    if constexpr (G == 1) {
        if (in) p.osum[s][e] = sum_rows(part + e, nc, ldp);
    } else {
        __shared__ double sh[G][W];
        const int64_t c0 = nc * y / G, c1 = nc * (y + 1) / G;
        sh[y][x] = in ? sum_rows(part + c0 * ldp + e, c1 - c0, ldp) : 0.;
        __syncthreads();
        if (y == 0 && in) {
            double o = sh[0][x];
#pragma unroll
            for (int k = 1; k < G; k++) o += sh[k][x];
            p.osum[s][e] = o;
        }
    }
}

// Per data point: weighted sub-exposure sums of the four sweeps in the
// reference's order (pb1f, pb1c, pb2f, pb2c, light_curve_comp.cpp:476-480),
// then third light.
__global__ void k_scatter(ScatterParams p, const double *__restrict__ o1f,
                          const double *__restrict__ o1c, const double *__restrict__ o2f,
                          const double *__restrict__ o2c, PhaseDev ph,
                          const DatumRec *__restrict__ data, const int64_t *__restrict__ off,
                          int32_t n, double *calc) {
    const int np = blockIdx.x * blockDim.x + threadIdx.x;
    if (np >= n) return;
    const int64_t e0 = off[np], e1 = e0 + (data[np].ndiv > 0 ? data[np].ndiv : 0);
    double c = 0.;
    for (int64_t e = e0; e < e1; e++)
        if (p.copy1 || ph.type[e] == 1) c += ph.w1[e] * o1f[e];
    if (!p.copy1)
        for (int64_t e = e0; e < e1; e++)
            if (ph.type[e] != 1) c += ph.w1[e] * o1c[e];
    double c2 = 0.;
    double *acc = p.fcomp ? &c2 : &c;  // iscale keeps the stars apart
    for (int64_t e = e0; e < e1; e++)
        if (p.copy2 || ph.type[e] == 3) *acc += ph.w2[e] * o2f[e];
    if (!p.copy2)
        for (int64_t e = e0; e < e1; e++)
            if (ph.type[e] != 3) *acc += ph.w2[e] * o2c[e];
    if (p.csum || p.fcomp) {
        // comp_disc / comp_edge / comp_spot of the point: sub-exposure sums
        // weighted and merged in order, over max(1, ndiv - 1)
        // (comp_light.cpp:323-408, light_curve_comp.cpp:476-490, 378-414)
        const DatumRec d = data[np];
        double phase, slfac;
        point_phase(p.pp, d, phase, slfac);
        const int ndiv = d.ndiv;
        double cd = 0.0, ce = 0.0, cs = 0.0;
        if (p.csum) {
            for (int nd = 0; nd < ndiv; nd++) {
                const int64_t e = e0 + nd;
                const double wgt = ndiv == 1 ? 1.0 : ((nd == 0 || nd == ndiv - 1) ? 0.5 : 1.0);
                cd += wgt * p.csum[e];
                ce += wgt * p.csum[p.ldc + e];
                cs += wgt * p.csum[2 * p.ldc + e];
            }
            const int norm = (ndiv - 1 > 1) ? ndiv - 1 : 1;
            cd /= norm;
            ce /= norm;
            cs /= norm;
        }
        if (p.fcomp) {
            double *f = p.fcomp + 5 * (int64_t)np;
            f[0] = c;
            f[1] = slfac * cd;
            f[2] = slfac * ce;
            f[3] = slfac * cs;
            f[4] = c2;
            calc[np] = 0.;
            return;
        }
        c += slfac * (cd + ce + cs);
    }
    calc[np] = c + p.third;
}

// Sums of K values over the 1024 threads of the block, in every thread: shuffles
// within the warps, then the 32 warps' sums the same way in each warp
// (deterministic; two barriers, where a tree in shared memory took ten for
// each value).
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; k++) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) sh[32 * k + w] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++) {
        v[k] = sh[32 * k + lane];
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    __syncthreads();
}
constexpr int kBlockSums = 32 * 4;  // doubles of shared memory for up to four values

// One block of 1024 threads: thread t takes points t, t+1024, ... in order,
// the block sums them in a fixed tree.
__device__ __forceinline__ void finalize_block(int32_t flags, const DatumRec *__restrict__ data,
                                               int32_t n, double *calc, double *sfac_io,
                                               double *out, double *sh) {
    const bool scale = flags & 1, rdata = flags & 2;
    const int t = threadIdx.x;
    if (scale) {
        double a = 0., b = 0., w = 0.;
        for (int i = t; i < n; i += 1024) {
            const DatumRec d = data[i];
            if (d.weight > 0.) {
                const double wgt = d.weight / sq(d.ferr);
                a += wgt * d.flux * calc[i];
                b += wgt * calc[i] * calc[i];
                w += d.weight;
            }
        }
        double s3[3] = {a, b, w};
        block_sums(s3, sh);
        const double sdy = s3[0], syy = s3[1], wnok = s3[2];
        const bool ok = wnok > 0.0;
        const double sc = ok ? sdy / syy : 1.;
        if (t == 0) {
            out[1] = wnok;
            for (int k = 0; k < 5; k++) sfac_io[k] = sc;
        }
        if (!ok) {
            if (t == 0) {
                out[0] = 0.;
                out[2] = 1.;
            }
            return;
        }
        for (int i = t; i < n; i += 1024) calc[i] = calc[i] * sc;
    } else {
        const double sc = sfac_io[0];
        for (int i = t; i < n; i += 1024) calc[i] *= sc;
        if (!rdata) {
            if (t == 0) out[2] = 0.;
            return;
        }
    }
    double cs = 0., w = 0.;
    for (int i = t; i < n; i += 1024) {
        const DatumRec d = data[i];
        if (d.weight > 0.) {
            cs += d.weight * sq((d.flux - calc[i]) / d.ferr);
            w += d.weight;
        }
    }
    double s2[2] = {cs, w};
    block_sums(s2, sh);
    if (t == 0) {
        out[0] = s2[0];
        if (!scale) out[1] = s2[1];
        out[2] = 1.;
    }
}

// What a call reads back besides the curve, gathered beside the finalize block:
// the diagnostic sums of the two stars' CTAs (k_continuum), the phase-0.5 sum of
// wdwarf and the device status.
__device__ __forceinline__ void tail_block(const TailIn &in, TailOut *out, double *sh) {
    const int t = threadIdx.x;
    for (int star = 0; star < 2; star++) {
        double v[4] = {0., 0., 0., 0.};
        const double *p = in.dsum[star];
        if (p)
            for (int64_t b = t; b < in.nb[star]; b += 1024)
#pragma unroll
                for (int k = 0; k < 4; k++) v[k] += p[4 * b + k];
        block_sums(v, sh);
        if (t < 4) out->diag[star][t] = t == 0 ? v[0] : t == 1 ? v[1] : t == 2 ? v[2] : v[3];
    }
    if (t == 0) {
        out->wsum = in.wsum ? *in.wsum : 0.;
        out->status = *in.status;
    }
}

__global__ void __launch_bounds__(1024) k_finalize(int32_t flags, const DatumRec *__restrict__ data,
                                                   int32_t n, double *calc, double sfac0,
                                                   TailIn in, TailOut *out) {
    __shared__ double sh[kBlockSums];
    if (blockIdx.x == 1) {
        tail_block(in, out, sh);
        return;
    }
    if (threadIdx.x == 0) out->sfac[0] = sfac0;
    __syncthreads();
    finalize_block(flags, data, n, calc, out->sfac, out->out, sh);
}

__global__ void __launch_bounds__(1024) k_tail(TailIn in, TailOut *out) {
    __shared__ double sh[kBlockSums];
    tail_block(in, out, sh);
}

// light_curve_comp_fast's interpolation (light_curve_comp_fast.cpp:46-83):
// point i takes the model at the sampled points around it (sample indices
// idx[0..m), ascending), linearly in time; with rdata, chi**2 and wnok over
// all points (out[0], out[1]). One block of 1024 threads, fixed-order tree.
__global__ void __launch_bounds__(1024) k_interp(const DatumRec *__restrict__ data, int32_t n,
                                                 const int64_t *__restrict__ idx, int32_t m,
                                                 const double *__restrict__ mc, double *calc,
                                                 int32_t rdata, double *out) {
    __shared__ double sh[kBlockSums];
    const int t = threadIdx.x;
    double cs = 0., w = 0.;
    for (int i = t; i < n; i += 1024) {
        int lo = 0, hi = m;  // first sample index >= i
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (idx[mid] < i) lo = mid + 1;
            else hi = mid;
        }
        double c;
        if (lo == 0) {
            c = mc[0];
        } else if (lo == m) {
            c = mc[m - 1];
        } else {
            const int64_t i1 = idx[lo - 1], i2 = idx[lo];
            const double tt = (data[i].time - data[i1].time) / (data[i2].time - data[i1].time);
            c = mc[lo - 1] * (1.0 - tt) + mc[lo] * tt;
        }
        calc[i] = c;
        const DatumRec d = data[i];
        if (d.weight > 0.) {
            w += d.weight;
            cs += d.weight * sq((d.flux - c) / d.ferr);
        }
    }
    if (!rdata) return;
    double s2[2] = {cs, w};
    block_sums(s2, sh);
    if (t == 0) {
        out[0] = s2[0];
        out[1] = s2[1];
    }
}

// Bounds of a group of consecutive lanes' faces (two per lane), W lanes a
// group: the mean of (nx, ny), the largest distance r from it and the extremes
// of cz. r and the extremes are widened well past FP32 rounding (1e-6, 1e-5).
// All-zero records (padding, faces with several ranges) add zeros whatever is
// concluded and are left out; a group of them alone gets cmax = -1. One with a face
// that is no finite number gets NaN: neither dark nor bright, its faces are tested singly.
template <int W>
__device__ __forceinline__ void group_mu(const float *nx, const float *ny, const float *cz,
                                         const bool *use, RunRec &R) {
    const unsigned full = 0xffffffffu;
    float sx = 0.f, sy = 0.f, cnt = 0.f;
    for (int k = 0; k < 2; k++)
        if (use[k]) {
            sx += nx[k] + 0.f * (nx[k] + ny[k] + cz[k]);
            sy += ny[k];
            cnt += 1.f;
        }
    for (int o = W / 2; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(full, sx, o);
        sy += __shfl_xor_sync(full, sy, o);
        cnt += __shfl_xor_sync(full, cnt, o);
    }
    const float ax = cnt > 0.f ? sx / cnt : 0.f, ay = cnt > 0.f ? sy / cnt : 0.f;
    float r = 0.f, hi = -2.f, lo = 2.f;
    for (int k = 0; k < 2; k++)
        if (use[k]) {
            r = fmaxf(r, sqrtf((nx[k] - ax) * (nx[k] - ax) + (ny[k] - ay) * (ny[k] - ay)));
            hi = fmaxf(hi, cz[k]);
            lo = fminf(lo, cz[k]);
        }
    for (int o = W / 2; o > 0; o >>= 1) {
        r = fmaxf(r, __shfl_xor_sync(full, r, o));
        hi = fmaxf(hi, __shfl_xor_sync(full, hi, o));
        lo = fminf(lo, __shfl_xor_sync(full, lo, o));
    }
    R.ax = ax;
    R.ay = ay;
    R.r = cnt > 0.f ? r * (1.f + 1e-6f) + 1e-6f : 0.f;
    R.cmax = cnt > 0.f ? hi + 1e-5f : -1.f;
    R.cmin = cnt > 0.f ? lo - 1e-5f : -1.f;
}

// The eclipse arcs of a group from its lanes' offsets off the reference phase
// ref (signed distances on the circle): hull [lo, hi), common part [lo2, hi2).
template <int W>
__device__ __forceinline__ void group_arcs(long long &lo, long long &hi, long long &lo2,
                                           long long &hi2, bool &whole, bool &bare) {
    const unsigned full = 0xffffffffu;
    for (int o = W / 2; o > 0; o >>= 1) {
        const long long a = __shfl_xor_sync(full, lo, o), b = __shfl_xor_sync(full, hi, o);
        const long long c = __shfl_xor_sync(full, lo2, o), d = __shfl_xor_sync(full, hi2, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
        lo2 = c > lo2 ? c : lo2;
        hi2 = d < hi2 ? d : hi2;
    }
    const unsigned lane = threadIdx.x & 31;
    const unsigned mine = W == 32 ? full : ((1u << W) - 1u) << (lane & ~(W - 1));
    whole = (__ballot_sync(full, whole) & mine) != 0u;
    bare = (__ballot_sync(full, bare) & mine) != 0u;
}

__device__ __forceinline__ void set_arcs(RunRec &R, unsigned long long ref, long long lo,
                                         long long hi, long long lo2, long long hi2, bool whole,
                                         bool bare) {
    R.hull = R.all = make_ulonglong2(0ull, 0ull);
    if (whole) {
        R.hull.y = ~0ull;
    } else if (hi > lo) {
        R.hull = make_ulonglong2(ref + (unsigned long long)lo,
                                 (unsigned long long)hi - (unsigned long long)lo);
        if (!bare && hi2 > lo2)
            R.all = make_ulonglong2(ref + (unsigned long long)lo2,
                                    (unsigned long long)hi2 - (unsigned long long)lo2);
    }
}

// The records of one run (RunRec), one warp per run, lane l holding pair l
// (normals, the z term cz, eclipse ranges): the four parts of 8 lanes first, then
// the run.
__device__ __forceinline__ void run_records(const float *nx, const float *ny, const float *cz,
                                            const bool *use, ulonglong2 *E, RunRec *out) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    RunRec part, whole_run;
    group_mu<8>(nx, ny, cz, use, part);
    group_mu<32>(nx, ny, cz, use, whole_run);
    // offsets from one range's start, as signed 64-bit distances on the circle;
    // ranges a quarter orbit long or further than that from it make the group's
    // hull "anywhere"; a live face without a range leaves no common part
    for (int k = 0; k < 2; k++)
        if (!use[k]) E[k].y = 0ull;
    const unsigned m = __ballot_sync(full, E[0].y != 0ull || E[1].y != 0ull);
    const unsigned long long mine = E[0].y != 0ull ? E[0].x : E[1].x;
    const unsigned long long ref = __shfl_sync(full, mine, m ? __ffs(m) - 1 : 0);
    constexpr long long kQuarter = 1ll << 62;
    if (!m) {  // most runs: no range to reduce
        set_arcs(part, 0ull, 0, 0, 0, 0, false, true);
        set_arcs(whole_run, 0ull, 0, 0, 0, 0, false, true);
        if ((lane & 7) == 0) out[1 + (lane >> 3)] = part;
        if (lane == 0) out[0] = whole_run;
        return;
    }
    long long lo = LLONG_MAX, hi = LLONG_MIN, lo2 = LLONG_MIN, hi2 = LLONG_MAX;
    bool whole = false, bare = false;
    for (int k = 0; k < 2; k++) {
        if (E[k].y == 0ull) {
            bare = bare || use[k];
            continue;
        }
        const long long off = (long long)(E[k].x - ref);
        if (E[k].y >= (unsigned long long)kQuarter || off >= kQuarter || off <= -kQuarter) {
            whole = true;
            continue;
        }
        const long long end = off + (long long)E[k].y;
        lo = off < lo ? off : lo;
        hi = end > hi ? end : hi;
        lo2 = off > lo2 ? off : lo2;
        hi2 = end < hi2 ? end : hi2;
    }
    long long l = lo, h = hi, l2 = lo2, h2 = hi2;
    bool w = whole, b = bare;
    group_arcs<8>(l, h, l2, h2, w, b);
    set_arcs(part, ref, l, h, l2, h2, w, b);
    group_arcs<32>(lo, hi, lo2, hi2, whole, bare);
    set_arcs(whole_run, ref, lo, hi, lo2, hi2, whole, bare);
    if ((lane & 7) == 0) out[1 + (lane >> 3)] = part;
    if (lane == 0) out[0] = whole_run;
}

// From the fast records: cz = cos(i) nz.
__device__ __forceinline__ void run_bound(const float *__restrict__ fp,
                                          const ulonglong2 *__restrict__ ecl, int64_t npairs,
                                          int64_t run, RunRec *out) {
    const int64_t q = run * 32 + (threadIdx.x & 31);
    float nx[2] = {0.f, 0.f}, ny[2] = {0.f, 0.f}, cz[2] = {0.f, 0.f};
    ulonglong2 E[2] = {make_ulonglong2(0ull, 0ull), make_ulonglong2(0ull, 0ull)};
    bool use[2] = {false, false};
    if (q < npairs) {
        const float4 P0 = reinterpret_cast<const float4 *>(fp)[4 * q];
        const float4 P1 = reinterpret_cast<const float4 *>(fp)[4 * q + 1];
        nx[0] = P0.x; nx[1] = P0.y; ny[0] = P0.z; ny[1] = P0.w; cz[0] = P1.x; cz[1] = P1.y;
        for (int k = 0; k < 2; k++) use[k] = nx[k] != 0.f || ny[k] != 0.f || cz[k] != 0.f;
        E[0] = ecl[2 * q];
        E[1] = ecl[2 * q + 1];
    }
    run_records(nx, ny, cz, use, E, out);
}

// From the general records (nx, ny, nz, flux) of n faces: cz = nz, the sweep
// multiplies by each entry's ez.
__global__ void k_run_bounds_geo(const float4 *__restrict__ geo,
                                 const ulonglong2 *__restrict__ ecl, int64_t n, RunRec *runs) {
    const int64_t run = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (run >= (n + kRunFaces - 1) / kRunFaces) return;  // whole warps
    const int64_t i = run * kRunFaces + 2 * (threadIdx.x & 31);
    float nx[2] = {0.f, 0.f}, ny[2] = {0.f, 0.f}, cz[2] = {0.f, 0.f};
    ulonglong2 E[2] = {make_ulonglong2(0ull, 0ull), make_ulonglong2(0ull, 0ull)};
    bool use[2] = {false, false};
    for (int k = 0; k < 2; k++) {
        if (i + k >= n) continue;
        const float4 g = geo[i + k];
        nx[k] = g.x; ny[k] = g.y; cz[k] = g.z;
        use[k] = g.x != 0.f || g.y != 0.f || g.z != 0.f;
        E[k] = ecl[i + k];
    }
    run_records(nx, ny, cz, use, E, runs + kRunRecs * run);
}

// From the FP64 columns: cz = nz; the arcs are drawn in (all) and out (hull) by
// two units, so that a phase is only ever decided by them where the sweep's
// double comparisons decide it alike.
__global__ void k_run_bounds64(FlatDev f) {
    const int64_t run = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (run >= (f.n + kRunFaces - 1) / kRunFaces) return;  // whole warps
    const int64_t i = run * kRunFaces + 2 * (threadIdx.x & 31), n0 = *f.n0;
    float nx[2] = {0.f, 0.f}, ny[2] = {0.f, 0.f}, cz[2] = {0.f, 0.f};
    ulonglong2 E[2] = {make_ulonglong2(0ull, 0ull), make_ulonglong2(0ull, 0ull)};
    bool use[2] = {false, false};
    for (int k = 0; k < 2; k++) {
        if (i + k >= f.n) continue;
        const double x = f.dx[i + k], y = f.dy[i + k], z = f.dz[i + k];
        use[k] = x != 0. || y != 0. || z != 0.;
        // vectors longer than one, or NaN, spoil their groups' bounds
        nx[k] = x * x + y * y + z * z < 1.000001 ? (float)x : nanf("");
        ny[k] = (float)y;
        cz[k] = (float)z;
        if (i + k < n0) continue;
        const double in = f.in1[i + k], out = f.out1[i + k];
        // ranges that a turn does not hold as they are: tested face by face
        E[k] = in >= 0. && in < 1. && out >= in ? ecl_fx64(in, out) : make_ulonglong2(0ull, ~0ull);
    }
    RunRec *out = f.runs + kRunRecs * run;
    run_records(nx, ny, cz, use, E, out);
    __syncwarp();
    const int r = threadIdx.x & 31;
    if (r < kRunRecs) {
        RunRec &R = out[r];
        if (R.hull.y != 0ull && R.hull.y != ~0ull) {
            R.hull.x -= 2ull;
            R.hull.y += 4ull;
        }
        if (R.all.y > 4ull) {
            R.all.x += 2ull;
            R.all.y -= 4ull;
        } else {
            R.all.y = 0ull;
        }
    }
}

__global__ void k_run_bounds(const float *__restrict__ fp, const ulonglong2 *__restrict__ ecl,
                             int64_t npairs, RunRec *runs) {
    const int64_t run = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (run >= (npairs + 31) / 32) return;  // whole warps
    run_bound(fp, ecl, npairs, run, runs + kRunRecs * run);
}

// Run records of the continuum list's slots (16 runs per 1024-face block).
__global__ void k_run_bounds_b(BatchDev b) {
    const int nk = b.counts[1];
    if (nk <= 0) return;
    const int64_t total = b.cont_blk[nk] * 16;
    const int64_t warps = (int64_t)gridDim.x * blockDim.x / 32;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < total;
         w += warps) {
        const int64_t B = w >> 4;
        const int k = find_seg(b.cont_blk, nk, B);
        const SlotDev &S = b.slots[b.cont_slot[k]];
        const int64_t run = (B - b.cont_blk[k]) * 16 + (w & 15);
        run_bound(b.fp + 8 * S.flat0, b.ecl + S.flat0, (S.nface + 1) / 2, run,
                  b.runs + kRunRecs * (S.flat0 / kRunFaces + run));
    }
}

// dst row r = src row rows[r] (rows of n doubles).
__global__ void k_gather_rows(const double *__restrict__ src, int32_t n,
                              const int32_t *__restrict__ rows, double *dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dst[(int64_t)blockIdx.y * n + i] = src[(int64_t)rows[blockIdx.y] * n + i];
}

// FP64 FlatGrid columns -> the packed mixed-precision view (used when a
// caller hands in a host FlatGrid through lcg_sum_star_multi).
__global__ void k_pack_flat(FlatDev f, int64_t n0, int need_pos) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i == 0) *f.n0 = n0;
    if (i >= f.n) return;
    f.geo[i] = make_float4((float)f.dx[i], (float)f.dy[i], (float)f.dz[i], (float)f.flux[i]);
    f.ecl[i] = i >= n0 ? ecl_fx64(f.in1[i], f.out1[i]) : make_ulonglong2(0ull, 0ull);
    if (need_pos) f.pos[i] = make_float4((float)f.px[i], (float)f.py[i], (float)f.pz[i], 0.f);
}

__global__ void k_pack_phases(PhaseDev ph) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ph.nent) return;
    ph.ef[e] = make_float4((float)ph.ex[e], (float)ph.ey[e], (float)ph.ez[e], 0.f);
    ph.pfx[e] = phase_fx64(ph.phin[e]);
}

// ---- batched stages ---------------------------------------------------------

// The slot's view of the batch point arrays.
__device__ __forceinline__ GridDev slot_grid(const GridDev &g, int64_t face0, int64_t nface,
                                             int64_t ntiled) {
    return GridDev{g.px + face0, g.py + face0, g.pz + face0, g.nx + face0, g.ny + face0,
                   g.nz + face0, g.area + face0, g.grav + face0, g.flux + face0, g.necl + face0,
                   g.ein + face0, g.eout + face0, nface, ntiled};
}

__global__ void __launch_bounds__(128) k_grid_b(BatchDev b) {
    const int nk = b.counts[0];
    if (nk <= 0) return;
    const int64_t total = b.geo_half[nk];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t u0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); u0 < total;
         u0 += stride) {
        int k = warp_search(nk, u0, [&](int i) { return b.geo_half[i]; });
        const SlotDev &S0 = b.slots[b.geo_slot[k]];
        const RingRec *rings = b.rings + S0.ring0;
        int lo = warp_search(S0.gp.nrings, u0 - b.geo_half[k],
                             [&](int i) { return (int64_t)rings[i].hoff; });
        const int64_t u = u0 + lane;
        if (u >= total) continue;
        while (u >= b.geo_half[k + 1]) {  // the warp reaches into the next slot: its first rings
            k++;
            lo = 0;
        }
        const SlotDev &S = b.slots[b.geo_slot[k]];
        grid_half(S.gp, b.rings + S.ring0, slot_grid(b.g, S.face0, S.nface, S.ntiled),
                  u - b.geo_half[k], lo, b.st + S.model);
    }
}

// Eclipsers whose reference sphere is at least this large share the front of
// the batch queue: a warp runs at its slowest lane's pace, and the boundaries of a
// white dwarf and of a larger star take different steps (ecl_root.cuh: the former
// have no gap to narrow). 256 models: bisections 3.84 ms so, 4.43 in queue order.
constexpr double kBigEclipser = 0.05;

// Sphere pre-test of the geometry list's faces; candidates are queued by
// their batch face index. Whole warps step together (queue_push votes).
__global__ void k_ecl_pre_b(BatchDev b) {
    const int nk = b.counts[0];
    if (nk <= 0) return;
    const int64_t total = b.geo_face[nk];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t u0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); u0 < total;
         u0 += stride) {
        const int64_t u = u0 + lane;
        bool cand = false, big = false;
        int32_t item = 0;
        int k = warp_search(nk, u0, [&](int i) { return b.geo_face[i]; });
        if (u < total) {
            while (u >= b.geo_face[k + 1]) k++;
            const SlotDev &S = b.slots[b.geo_slot[k]];
            const int64_t i = u - b.geo_face[k];
            cand = ecl_pre_face<false>(S.ep, S.eclipse_on, slot_grid(b.g, S.face0, S.nface, S.ntiled), i);
            item = (int32_t)(S.face0 + i);
            big = S.ep.comp_rref >= kBigEclipser;
        }
        // eclipses by a large star to the front of the queue, by a white dwarf to
        // the back
        const unsigned back = __ballot_sync(0xffffffffu, cand && !big);
        queue_push(cand && big, item, b.queue, b.counters);
        if (back) {
            const int leader = __ffs(back) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(&b.counters[4], __popc(back));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (cand && !big)
                b.queue[b.qcap - 1 - (base + __popc(back & ((1u << lane) - 1u)))] = item;
        }
    }
}

// After k_ecl_pre_b: the candidate count covers both ends of the queue;
// counters[5] keeps the front's.
__global__ void k_ecl_join_b(BatchDev b) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        b.counters[5] = b.counters[0];
        b.counters[0] += b.counters[4];
    }
}

// Candidate k of the batch queue (front, then back in push order).
__device__ __forceinline__ int32_t queue_at(const BatchDev &b, int k) {
    const int front = b.counters[5];
    return k < front ? b.queue[k] : b.queue[b.qcap - 1 - (k - front)];
}

// k_ecl_roche over the batch queue: each candidate finds its slot by its
// face index.
__device__ __forceinline__ bool batch_warp_mode(const BatchDev &b, int32_t warp_max) {
    return b.counters[0] <= warp_max;
}

__global__ void __launch_bounds__(128, 4) k_ecl_roche_b(BatchDev b, int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = b.counters[0];
    const GridDev g = b.g;
    if (batch_warp_mode(b, warp_max)) {
        for (;;) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&b.counters[1], 1);
            k = __shfl_sync(full, k, 0);
            if (k >= total) break;
            const int32_t i = queue_at(b, k);
            const SlotDev &S = b.slots[find_seg(b.face0, b.nslots, i)];
            const EclParams &p = S.ep;
            const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
            double ing = 0., egr = 0.;
            int s = 0;
            const bool ecl = ingress_egress_warp(p.comp_star, p.q, p.comp_spin, p.cosi, p.sini,
                                                 p.delta, pos, p.comp_rref, p.comp_pref, ing,
                                                 egr, s);
            if (lane == 0) {
                if (s) {
                    set_status(b.st + S.model, s, i - S.face0);
                } else if (ecl) {
                    g.necl[i] = 1;
                    g.ein[i] = ing;
                    g.eout[i] = egr;
                }
            }
        }
        return;
    }
}

// Thread mode of the batched eclipse, in two passes whose code is small enough
// to stay in the instruction cache (the fused solve stalled on instruction
// fetch): the sphere test and pot_min per candidate, then the ingress and
// egress bisections (ingress_egress.cpp:61-86) on the two lanes of a pair.
// Warps take consecutive candidates (similar iteration counts run together).
// Same arithmetic and decisions as ingress_egress: identical results.
__global__ void __launch_bounds__(128, 4) k_ecl_potmin_b(BatchDev b, int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = b.counters[0];
    if (batch_warp_mode(b, warp_max)) return;
    const GridDev g = b.g;
    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&b.counters[2], 32);
        base = __shfl_sync(full, base, 0);
        if (base >= total) break;
        const int k = base + lane;
        bool hit = false;
        if (k < total) {
            const int32_t i = queue_at(b, k);
            const SlotDev &S = b.slots[find_seg(b.face0, b.nslots, i)];
            const EclParams &p = S.ep;
            const V3 pos = v3(g.px[i], g.py[i], g.pz[i]);
            const V3 cofm = p.comp_star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
            double phi1, phi2, lam1, lam2, phi = 0., lam = 0.;
            if (sphere_eclipse_ph(p.cosi, p.sini, pos, cofm, p.comp_rref, phi1, phi2, lam1,
                                  lam2)) {
                const double ACC = 2. * sqrt(2. * kTwoPi * (lam2 - lam1) * p.delta);
                int s = 0;
                hit = pot_min(p.comp_star, p.q, p.comp_spin, p.cosi, p.sini, pos, phi1, phi2,
                              lam1, lam2, p.comp_rref, p.comp_pref, ACC, phi, lam, s);
                if (s) {
                    set_status(b.st + S.model, s, i - S.face0);
                    hit = false;
                }
                b.es[k] = make_double4(phi, phi1, phi2, ACC);
            }
        }
        push_hits(hit, k, b.hits, &b.counters[6]);
    }
}

// 4 blocks of 4 warps per SM (bisect_blocks_per_sm; the registers of 6 spill, 8.41 ms at 4
// and 8.36 at 6 for two batches of 256 models, 4 faster on small ones)
template <int NB>
__global__ void __launch_bounds__(128, NB)
    k_ecl_bisect_b(__grid_constant__ const BatchDev b, int32_t warp_max) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = b.counters[0];
    if (batch_warp_mode(b, warp_max)) return;
    const int64_t n2 = 2 * (int64_t)b.counters[6];
    for (;;) {
        int64_t base = 0;
        if (lane == 0) base = atomicAdd(&b.counters[3], 32);
        base = __shfl_sync(full, base, 0);
        if (base >= n2) break;
        const int64_t u = base + lane;
        const int side = (int)(u & 1);
        const bool live = u < n2;
        const int k = live ? b.hits[u >> 1] : 0;
        const int32_t i = live ? queue_at(b, k) : 0;
        const int sl = find_seg(b.face0, b.nslots, i);
        const double4 E = live ? b.es[k] : make_double4(0., 0., 0., 0.);
        const V3 pos = live ? v3(b.g.px[i], b.g.py[i], b.g.pz[i]) : v3(0., 0., 0.);
        int s = 0;
        double v = bisect_warp(b.slots[sl].ep, live, E.x, side ? E.z : E.y, E.w, pos, s);
        v = v - floor(v);
        const double other = __shfl_xor_sync(full, v, 1);
        const int os = __shfl_xor_sync(full, s, 1);
        if (live && side == 0) {
            const SlotDev &S = b.slots[sl];
            if (s || os) {
                set_status(b.st + S.model, s ? s : os, i - S.face0);
            } else {
                double egr = other;
                if (egr < v) egr++;
                b.g.necl[i] = 1;
                b.g.ein[i] = v;
                b.g.eout[i] = egr;
            }
        }
    }
}

// Partition counts per 1024-face block of the geometry list's slots, a warp per
// block. They change with the eclipses only, so they stand until the slot's
// geometry is rebuilt, as do the slot's offsets (k_flat_scan_b) and ranges.
__global__ void __launch_bounds__(256) k_flat_count_b(BatchDev b) {
    const int nk = b.counts[0];
    if (nk <= 0) return;
    const int64_t total = b.geo_blk[nk], warps = (int64_t)gridDim.x * 8;
    const int lane = threadIdx.x & 31;
    for (int64_t B = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5; B < total; B += warps) {
        const int k = find_seg(b.geo_blk, nk, B);
        const SlotDev &S = b.slots[b.geo_slot[k]];
        const int64_t lb = B - b.geo_blk[k];
        const uint8_t *necl = b.g.necl + S.face0 + lb * kFlatBlock;
        const int left = (int)(S.nface - lb * kFlatBlock < kFlatBlock ? S.nface - lb * kFlatBlock
                                                                      : kFlatBlock);
        int c = 0;
#pragma unroll 8
        for (int i = lane; i < kFlatBlock; i += 32)
            c += __popc(__ballot_sync(0xffffffffu, i < left && necl[i] == 1));
        if (lane == 0) b.blockcnt[S.blk0 + lb] = c;
    }
}

__global__ void __launch_bounds__(1024) k_flat_scan_b(BatchDev b) {
    const int nk = b.counts[0];
    for (int k = blockIdx.x; k < nk; k += gridDim.x) {
        const int s = b.geo_slot[k];
        const SlotDev &S = b.slots[s];
        const int32_t nb = (int32_t)((S.nface + kFlatBlock - 1) / kFlatBlock);
        scan_blocks(b.blockcnt + S.blk0, nb, S.nface, b.n0 + s);
    }
}

// Continuum and stable partition into fast sweep records in one pass, a CTA per
// 1024-face block of the continuum list's slots: each face's record is formed
// from its point once (57 B read, 81 with a range) and goes to its place among
// the block's never-eclipsed or one-range faces in shared memory; the two
// segments are then written out in the pair layout, consecutive floats by
// consecutive threads. Separate passes wrote the fluxes and read the normals
// again, and scattered 4-byte stores 8 bytes apart: 256 models (24.7 M faces)
// 1.47 ms for the continuum, the counts and the records together -> 0.72. Eclipse ranges
// are written for rebuilt geometry only. The record after an odd last face is
// zeroed (the sweep reads faces in pairs).
constexpr int kRecPad = kFlatBlock + 4;  // the eight quantities of a face in different banks
constexpr size_t kContSmem = 8 * (size_t)kRecPad * sizeof(float) + kFlatBlock * sizeof(ulonglong2);

__global__ void __launch_bounds__(256) k_cont_flat_b(BatchDev b) {
    extern __shared__ __align__(16) unsigned char cont_smem[];
    ulonglong2 *secl = reinterpret_cast<ulonglong2 *>(cont_smem);
    float *rec = reinterpret_cast<float *>(secl + kFlatBlock);
    __shared__ int32_t before[32], ones;
    const int nk = b.counts[1];
    if (nk <= 0) return;
    const int64_t total = b.cont_blk[nk];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int64_t B = blockIdx.x; B < total; B += gridDim.x) {
        const int k = find_seg(b.cont_blk, nk, B);
        const int s = b.cont_slot[k];
        const SlotDev &S = b.slots[s];
        const int64_t lb = B - b.cont_blk[k], i0 = lb * kFlatBlock, n = S.nface;
        const GridDev g = slot_grid(b.g, S.face0, n, S.ntiled);
        const int in_block = (int)(n - i0 < kFlatBlock ? n - i0 : kFlatBlock);
        // ranks of the one-range faces: ballots, then a scan over the 32 warp slices
        unsigned m[4];
#pragma unroll
        for (int it = 0; it < 4; it++) {
            const int i = it * 256 + t;
            m[it] = __ballot_sync(0xffffffffu, i < in_block && g.necl[i0 + i] == 1);
            if (lane == 0) before[it * 8 + w] = __popc(m[it]);
        }
        __syncthreads();
        if (t < 32) {
            const int v = before[t];
            int x = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            before[t] = x - v;
            if (t == 31) ones = x;
        }
        __syncthreads();
        const int n1 = ones, n0l = in_block - n1;
        const FastCoef &fc = S.fc;
        const bool fresh = S.fresh != 0;
#pragma unroll 1
        for (int it = 0; it < 4; it++) {
            const int i = it * 256 + t;
            if (i >= in_block) break;
            const bool flag = (m[it] >> lane) & 1u;
            const int rank1 = before[it * 8 + w] + __popc(m[it] & ((1u << lane) - 1u));
            const int at = flag ? n0l + rank1 : i - rank1;
            const double fl = (double)continuum_flux(S.cp, g, i0 + i);
            rec[at] = (float)g.nx[i0 + i];
            rec[kRecPad + at] = (float)g.ny[i0 + i];
            rec[2 * kRecPad + at] = (float)(fc.cosi * g.nz[i0 + i]);
#pragma unroll
            for (int q = 0; q < 5; q++) rec[(3 + q) * kRecPad + at] = (float)(fl * fc.p[q]);
            if (fresh && flag) secl[rank1] = ecl_fx64(g.ein[i0 + i], g.eout[i0 + i]);
        }
        __syncthreads();
        float *fp = b.fp + 8 * S.flat0;
        ulonglong2 *ecl = b.ecl + S.flat0;
        const int64_t boff = b.blockcnt[S.blk0 + lb];
#pragma unroll
        for (int seg = 0; seg < 2; seg++) {
            const int64_t d = seg ? b.n0[s] + boff : i0 - boff;
            const int count = seg ? n1 : n0l, o = seg ? n0l : 0;
            // floats of the pairs the segment touches; dest = d + j
            const int64_t a0 = 16 * (d >> 1), a1 = 16 * ((d + count + 1) >> 1);
            for (int64_t a = a0 + t; a < a1; a += 256) {
                const int j = (int)(2 * (a >> 4) + (a & 1) - d);
                if (j >= 0 && j < count) fp[a] = rec[(int)((a & 15) >> 1) * kRecPad + o + j];
            }
            if (fresh)
                for (int j = t; j < count; j += 256)
                    ecl[d + j] = seg ? secl[j] : make_ulonglong2(0ull, 0ull);
        }
        if ((n & 1) && i0 + in_block == n) {
            if (t < 8) fp[16 * (n >> 1) + 1 + 2 * t] = 0.f;
            if (t == 8) ecl[n] = make_ulonglong2(0ull, 0ull);
        }
        __syncthreads();
    }
}

__global__ void k_phases_b(BatchDev b, const DatumRec *__restrict__ data,
                           const int64_t *__restrict__ off, int32_t n, BatchPhases ph) {
    const int np = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y;
    if (np >= n || !b.models[m].live) return;
    const PhaseParams &p = b.models[m].pp;
    const DatumRec d = data[np];
    double phase, slfac;
    point_phase(p, d, phase, slfac);
    const double expose = d.expose / p.period;
    const int ndiv = d.ndiv;
    const double norm = (ndiv - 1 > 1) ? ndiv - 1 : 1;
    int64_t e = m * ph.ldp + off[np];
    for (int nd = 0; nd < ndiv; ++nd, ++e) {
        double phi, wgt;
        sub_exposure(phase, expose, ndiv, nd, phi, wgt);
        const V3 earth = set_earth(p.cosi, p.sini, phi);
        const double phin = phi - floor(phi);
        ph.w1[e] = slfac * wgt * gi_scale1(p.gi, phi) / norm;
        ph.w2[e] = slfac * wgt * gi_scale2(p.gi, phi) / norm;
        ph.ef[e] = make_float4((float)earth.x, (float)earth.y, (float)earth.z, 0.f);
        ph.pfx[e] = phase_fx64(phin);
    }
}

// Chunk partials of each slot summed in chunk order, per phase entry.
__global__ void k_reduce_b(BatchDev b, const double *__restrict__ part, int64_t ldp, int64_t nent,
                           double *osum) {
    const int s = blockIdx.y;
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nent || !b.slots[s].live) return;
    const int64_t c0 = b.chunk_pre[s], c1 = b.chunk_pre[s + 1];
    osum[s * ldp + e] = sum_rows(part + c0 * ldp + e, c1 - c0, ldp);
}

// Per model and point: star 1 then star 2 sub-exposure sums, third light.
__global__ void k_scatter_b(BatchDev b, BatchPhases ph, const double *__restrict__ osum,
                            const DatumRec *__restrict__ data, const int64_t *__restrict__ off,
                            int32_t n, double *calc) {
    const int np = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y;
    if (np >= n || !b.models[m].live) return;
    const int64_t row = m * ph.ldp;
    const double *o1 = osum + (2 * (int64_t)m) * ph.ldp, *o2 = o1 + ph.ldp;
    const int64_t e0 = off[np], e1 = e0 + (data[np].ndiv > 0 ? data[np].ndiv : 0);
    double c = 0.;
    for (int64_t e = e0; e < e1; e++) c += ph.w1[row + e] * o1[e];
    for (int64_t e = e0; e < e1; e++) c += ph.w2[row + e] * o2[e];
    calc[m * (int64_t)n + np] = c + b.models[m].third;
}

__global__ void __launch_bounds__(1024) k_finalize_b(BatchDev b, int32_t flags,
                                                     const DatumRec *__restrict__ data,
                                                     int32_t n, double *calc, double *sfac,
                                                     double *out) {
    __shared__ double sh[kBlockSums];
    const int m = blockIdx.x;
    if (!b.models[m].live) return;  // keeps the previous call's results
    double *sf = sfac + 5 * (int64_t)m;
    if (threadIdx.x == 0) sf[0] = b.models[m].sfac0;
    __syncthreads();
    finalize_block(flags, data, n, calc + m * (int64_t)n, sf, out + 3 * (int64_t)m, sh);
}

inline unsigned nblocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_pack_flat(FlatDev f, int64_t n0, int need_pos, cudaStream_t s) {
    k_pack_flat<<<nblocks(f.n > 0 ? f.n : 1, 256), 256, 0, s>>>(f, n0, need_pos);
    count_launch();
}

void launch_pack_phases(PhaseDev ph, cudaStream_t s) {
    if (ph.nent <= 0) return;
    k_pack_phases<<<nblocks(ph.nent, 256), 256, 0, s>>>(ph);
    count_launch();
}

void launch_grid(const GridParams &p, const RingRec *rings, GridDev g, int32_t *counters,
                 DevStatus *st, cudaStream_t s) {
    if (p.nhalf <= 0) return;
    k_grid<<<nblocks(p.nhalf, 128), 128, 0, s>>>(p, rings, g, counters, st);
    count_launch();
}

// Resident blocks of 128 threads per SM for the bisection kernels: 4 (no
// register spills, 128 registers a thread) or 6 (80 registers, a few
// spills, more warps to hide FP64 latency); LCG_ECL_BISECT_BLOCKS=6 selects
// the second, for measurement.
int bisect_blocks_per_sm() {
    static const int nb = [] {
        const char *v = getenv("LCG_ECL_BISECT_BLOCKS");
        return (v && atoi(v) == 6) ? 6 : 4;
    }();
    return nb;
}

void launch_eclipse(const EclParams &p, int32_t eclipse_on, GridDev g, int32_t *queue,
                    int32_t *counters, double4 *es, int32_t *hits, DevStatus *st, int nsm,
                    int32_t warp_mode, cudaStream_t s) {
    if (g.n <= 0) return;
    // two lanes per face at four CTAs of 128 per SM
    if (eclipse_on && p.comp_roche && warp_mode <= 0 && g.n <= (int64_t)nsm * 256) {
        k_ecl_small<<<nblocks(2 * g.n, 128), 128, 0, s>>>(p, eclipse_on, g, st);
        count_launch();
        return;
    }
    k_ecl_pre<<<nblocks(g.n, 256), 256, 0, s>>>(p, eclipse_on, g, queue, counters);
    count_launch();
    if (eclipse_on && p.comp_roche) {
        // 4 blocks of 4 warps per SM; no more warps than faces
        unsigned nb = (unsigned)nsm * 4u;
        const unsigned need = nblocks(g.n, 4);
        if (need < nb) nb = need;
        // warp mode on request only: with the boundary's root found first, the
        // thread mode has the shorter latency for any number of candidates
        const int32_t warp_max = warp_mode > 0 ? warp_mode : -1;
        if (warp_max > 0) {
            k_ecl_roche<<<nb, 128, 0, s>>>(p, g, queue, counters, st, warp_max);
            count_launch();
        }
        k_ecl_potmin<<<nb, 128, 0, s>>>(p, g, queue, counters, es, hits, st, warp_max);
        count_launch();
        const int nbs = bisect_blocks_per_sm();
        const unsigned cap = (unsigned)nsm * (unsigned)nbs;
        const unsigned nbb = need < cap ? need : cap;
        if (nbs == 6)
            k_ecl_bisect<6><<<nbb, 128, 0, s>>>(p, g, queue, counters, es, hits, st, warp_max);
        else
            k_ecl_bisect<4><<<nbb, 128, 0, s>>>(p, g, queue, counters, es, hits, st, warp_max);
        count_launch();
    }
}

int64_t cont_blocks(int64_t n) { return (n + kContBlock - 1) / kContBlock; }

void launch_continuum(const ContParams &p, GridDev g, int32_t *cnt, double *dsum,
                      cudaStream_t s) {
    if (g.n <= 0) return;
    k_continuum<<<(unsigned)cont_blocks(g.n), kContBlock, 0, s>>>(p, g, cnt, dsum);
    count_launch();
}

void launch_flatten(GridDev g, FlatDev f, const int32_t *cnt, int mixed, int need_pos,
                    const FastCoef &fc, cudaStream_t s) {
    if (g.n <= 0) {
        cudaMemsetAsync(f.n0, 0, 2 * sizeof(int64_t), s);
        return;
    }
    const int64_t cover = mixed && fc.on ? f.npad : g.n;
    k_flat_scatter<<<nblocks(cover, kFlatBlock), kFlatBlock, 0, s>>>(
        g, f, cnt, (int32_t)cont_blocks(g.n), mixed, need_pos, fc);
    count_launch();
    if (mixed && fc.on) launch_run_bounds(f.fp, f.ecl, f.npad / 2, f.runs, s);
    else if (mixed) launch_run_bounds_geo(f, s);
    else launch_run_bounds64(f, s);
}

void launch_phases(const PhaseParams &p, const DatumRec *data, const int64_t *off, int32_t n,
                   PhaseDev ph, bool extra, V3 ew, double phw, cudaStream_t s) {
    if (n <= 0) return;
    k_phases<<<nblocks(n + (extra ? 1 : 0), 128), 128, 0, s>>>(p, data, off, n, ph, extra, ew, phw);
    count_launch();
}

void launch_scatter(const ScatterParams &p, const ReduceParams &r, const PhaseDev &ph,
                    const DatumRec *data, const int64_t *off, int32_t n, double *calc,
                    cudaStream_t s) {
    if (n <= 0) return;
    int64_t nmax = 0;
    for (int k = 0; k < 4; k++)
        if (r.part[k] && r.nent[k] > nmax) nmax = r.nent[k];
    if (nmax > 0) {
        if (r.in_order) k_reduce_chunks<1><<<dim3(nblocks(nmax, 256), 4), 256, 0, s>>>(r);
        else k_reduce_chunks<8><<<dim3(nblocks(nmax, 32), 4), 256, 0, s>>>(r);
        count_launch();
    }
    k_scatter<<<nblocks(n, 128), 128, 0, s>>>(p, r.osum[0], r.osum[1], r.osum[2], r.osum[3], ph,
                                              data, off, n, calc);
    count_launch();
}

void launch_finalize(int32_t flags, const DatumRec *data, int32_t n, double *calc, double sfac0,
                     const TailIn &in, TailOut *out, cudaStream_t s) {
    k_finalize<<<2, 1024, 0, s>>>(flags, data, n, calc, sfac0, in, out);
    count_launch();
}

void launch_tail(const TailIn &in, TailOut *out, cudaStream_t s) {
    k_tail<<<1, 1024, 0, s>>>(in, out);
    count_launch();
}

void launch_interp(const DatumRec *data, int32_t n, const int64_t *idx, int32_t m,
                   const double *mc, double *calc, int32_t rdata, double *out, cudaStream_t s) {
    if (n <= 0 || m <= 0) return;
    k_interp<<<1, 1024, 0, s>>>(data, n, idx, m, mc, calc, rdata, out);
    count_launch();
}

void launch_run_bounds(const float *fp, const ulonglong2 *ecl, int64_t npairs, RunRec *runs,
                       cudaStream_t s) {
    const int64_t nruns = (npairs + 31) / 32;
    if (nruns <= 0) return;
    k_run_bounds<<<nblocks(nruns * 32, 256), 256, 0, s>>>(fp, ecl, npairs, runs);
    count_launch();
}

void launch_run_bounds_geo(const FlatDev &f, cudaStream_t s) {
    const int64_t nruns = (f.n + kRunFaces - 1) / kRunFaces;
    if (nruns <= 0) return;
    k_run_bounds_geo<<<nblocks(nruns * 32, 256), 256, 0, s>>>(f.geo, f.ecl, f.n, f.runs);
    count_launch();
}

void launch_run_bounds64(const FlatDev &f, cudaStream_t s) {
    const int64_t nruns = (f.n + kRunFaces - 1) / kRunFaces;
    if (nruns <= 0) return;
    k_run_bounds64<<<nblocks(nruns * 32, 256), 256, 0, s>>>(f);
    count_launch();
}

void launch_batch_run_bounds(const BatchDev &b, int nsm, cudaStream_t s) {
    k_run_bounds_b<<<nsm * 8, 256, 0, s>>>(b);
    count_launch();
}

void launch_gather_rows(const double *src, int32_t n, const int32_t *rows, int32_t count,
                        double *dst, cudaStream_t s) {
    if (n <= 0 || count <= 0) return;
    k_gather_rows<<<dim3(nblocks(n, 256), (unsigned)count), 256, 0, s>>>(src, n, rows, dst);
    count_launch();
}

// ---- batched launchers -------------------------------------------------------

void launch_batch_grid(const BatchDev &b, int nsm, cudaStream_t s) {
    // one wave of the blocks that fit (its registers allow 5 of 128 threads per
    // SM): a grid-stride loop over more blocks than fit runs a second, partial
    // wave after the first
    static const int per_sm = [] {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_grid_b, 128, 0) != cudaSuccess ||
            nb < 1)
            nb = 4;
        return nb;
    }();
    k_grid_b<<<nsm * per_sm, 128, 0, s>>>(b);
    count_launch();
}

void launch_batch_eclipse(const BatchDev &b, int nsm, int32_t warp_mode, cudaStream_t s) {
    cudaMemsetAsync(b.counters, 0, 8 * sizeof(int32_t), s);
    k_ecl_pre_b<<<nsm * 4, 256, 0, s>>>(b);
    count_launch();
    k_ecl_join_b<<<1, 32, 0, s>>>(b);
    count_launch();
    const int32_t warp_max = warp_mode > 0 ? warp_mode : -1;
    if (warp_max > 0) {
        k_ecl_roche_b<<<nsm * 4, 128, 0, s>>>(b, warp_max);
        count_launch();
    }
    k_ecl_potmin_b<<<nsm * 4, 128, 0, s>>>(b, warp_max);
    count_launch();
    if (bisect_blocks_per_sm() == 6)
        k_ecl_bisect_b<6><<<nsm * 6, 128, 0, s>>>(b, warp_max);
    else
        k_ecl_bisect_b<4><<<nsm * 4, 128, 0, s>>>(b, warp_max);
    count_launch();
}

void launch_batch_partition(const BatchDev &b, int nsm, cudaStream_t s) {
    k_flat_count_b<<<nsm * 8, 256, 0, s>>>(b);
    count_launch();
    k_flat_scan_b<<<nsm, 1024, 0, s>>>(b);
    count_launch();
}

void launch_batch_continuum(const BatchDev &b, int nsm, cudaStream_t s) {
    cudaFuncSetAttribute(k_cont_flat_b, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kContSmem);
    k_cont_flat_b<<<nsm * 4, 256, kContSmem, s>>>(b);
    count_launch();
    launch_batch_run_bounds(b, nsm, s);
}

void launch_batch_phases(const BatchDev &b, const DatumRec *data, const int64_t *off, int32_t n,
                         const BatchPhases &ph, cudaStream_t s) {
    if (n <= 0 || b.nmodels <= 0) return;
    k_phases_b<<<dim3(nblocks(n, 128), (unsigned)b.nmodels), 128, 0, s>>>(b, data, off, n, ph);
    count_launch();
}

void launch_batch_reduce(const BatchDev &b, const BatchPhases &ph, const double *part,
                         int64_t ldp, double *osum, const DatumRec *data, const int64_t *off,
                         int32_t n, int32_t flags, double *calc, double *sfac, double *out,
                         cudaStream_t s) {
    if (n <= 0 || b.nmodels <= 0) return;
    if (ph.nent > 0) {
        k_reduce_b<<<dim3(nblocks(ph.nent, 256), (unsigned)b.nslots), 256, 0, s>>>(
            b, part, ldp, ph.nent, osum);
        count_launch();
    }
    k_scatter_b<<<dim3(nblocks(n, 128), (unsigned)b.nmodels), 128, 0, s>>>(b, ph, osum, data,
                                                                             off, n, calc);
    count_launch();
    k_finalize_b<<<b.nmodels, 1024, 0, s>>>(b, flags, data, n, calc, sfac, out);
    count_launch();
}

}  // namespace lcg
