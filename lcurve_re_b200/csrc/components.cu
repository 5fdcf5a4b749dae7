// components.cu — accretion disc, disc rim and bright spot; iscale fits.
//
// Element kernels restate set_disc_grid (set_disc_grid.cpp:27-127), the
// outer rim of set_disc_edge (:144-264), set_bright_spot_grid
// (set_bright_spot_grid.cpp:27-100), their continua (set_disc_continuum.cpp)
// and star_eclipse (star_eclipse.cpp:15-26) with one thread per element: the
// per-ring and per-model scalars come from the host, the trigonometry, the
// continuum and the eclipse solves run on the device. Element sums per phase
// entry follow comp_disc / comp_edge / comp_spot (comp_light.cpp:323-408) with
// the elements in vector order, summed in chunks of 256 whose partial sums
// are added in order (the reference's single serial sum, regrouped: equal to
// rounding). Compiled with --fmad=false.
#include "context.h"
#include "eclipse.cuh"
#include "fixed_phase.cuh"
#include "flux_groups.cuh"

namespace lcg {

namespace {

constexpr int kThreadsC = 128;

__device__ __forceinline__ void report(DevStatus *st, int code, int idx) {
    if (atomicCAS(&st->code, 0, code) == 0) st->face = idx;
}

// Component elements report -(1 + element index) so that the host can tell
// them from star faces.
__device__ __forceinline__ int elem_tag(int i) { return -1 - i; }

// The boundary `side` (0 ingress, 1 egress) of the eclipse of posn by star 1
// or 2 (ingress_egress.cpp:35-97), by every lane of a warp at once: ecl whether
// it is eclipsed at all, at the phase; s the failure of pot_min or of this side.
__device__ __forceinline__ void elem_boundary(const CompParams &p, int star, int side, bool on,
                                              V3 posn, bool &ecl, double &at, int &s) {
    const EclParams &E = p.ecl[star];
    double phi1 = 0., phi2 = 0., lam1, lam2, phi = 0., lam, acc = 0.;
    ecl = false;
    at = 0.;
    s = 0;
    bool live = false;
    if (on) {
        const V3 c = star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
        const double rs = E.comp_roche ? E.comp_rref : E.comp_r;
        ecl = sphere_eclipse_ph(E.cosi, E.sini, posn, c, rs, phi1, phi2, lam1, lam2);
        if (ecl && E.comp_roche) {
            acc = 2. * sqrt(2. * kTwoPi * (lam2 - lam1) * E.delta);
            ecl = live = pot_min(star, E.q, E.comp_spin, E.cosi, E.sini, posn, phi1, phi2, lam1,
                                 lam2, E.comp_rref, E.comp_pref, acc, phi, lam, s);
        }
    }
    at = side ? phi2 : phi1;
    const double v = bisect_warp(E, live, phi, at, acc, posn, s);
    if (live) at = v - floor(v);
}

// The eclipses of one element from its four lanes (star 1 ingress, egress, star 2
// ingress, egress): the opaque disc's (disc and rim only; the spot gets none,
// set_bright_spot_grid.cpp:80-81), then star 1's, then star 2's
// (set_disc_grid.cpp:99-113). trap1: a Roche_Error from star 1 becomes the
// range (0, 1), as for the rim's upper elements (set_disc_grid.cpp:222-231).
// Nearly every disc element is a candidate of the donor, and the solves are
// serial FP64 chains: a lane per boundary runs the four side by side. 13,500
// disc, rim and spot elements: 427 us with one thread solving all of an
// element's eclipses by bisection -> 75 us.
__device__ void elem_eclipses(const CompParams &p, V3 posn, bool in_range, bool opaque, bool trap1,
                              ElemRec &r, DevStatus *st, int idx) {
    const unsigned full = 0xffffffffu;
    const int sub = threadIdx.x & 3;
    bool ecl;
    double at;
    int s;
    elem_boundary(p, sub >> 1, sub & 1, in_range && (sub < 2 ? p.eclipse1 : p.eclipse2), posn, ecl,
                  at, s);
    // lane 0 of the element collects (a failure of the ingress comes first)
    bool necl[2];
    double in[2], out[2];
    int es[2];
    for (int k = 0; k < 2; k++) {
        const int src = (threadIdx.x & 28) + 2 * k;
        necl[k] = __shfl_sync(full, ecl, src);
        in[k] = __shfl_sync(full, at, src);
        out[k] = __shfl_sync(full, at, src + 1);
        const int s0 = __shfl_sync(full, s, src), s1 = __shfl_sync(full, s, src + 1);
        es[k] = s0 ? s0 : s1;
        if (p.ecl[k].comp_roche && out[k] < in[k]) out[k]++;
    }
    if (!in_range || sub != 0) return;
    r.nr = 0;  // an element whose eclipse failed is left with none
    for (int k = 0; k < kMaxRanges; k++) r.r[k] = make_double2(0., 0.);
    int nr = 0;
    double rin[kMaxRanges], rout[kMaxRanges];
    if (opaque) {
        int ds = 0;
        disc_eclipse(p.dg, posn, nr, rin, rout, kMaxRanges, ds);
        if (ds) { report(st, ds, idx); return; }
    }
    for (int k = 0; k < 2; k++) {
        if (es[k]) {
            if (!(k == 0 && trap1 && es[k] == kEclRoche)) { report(st, es[k], idx); return; }
            necl[k] = true;
            in[k] = 0.;
            out[k] = 1.;
        }
        if (necl[k]) {
            if (nr < kMaxRanges) { rin[nr] = in[k]; rout[nr] = out[k]; }
            nr++;
        }
    }
    r.nr = nr < kMaxRanges ? nr : kMaxRanges;
    for (int k = 0; k < kMaxRanges; k++)
        r.r[k] = k < r.nr ? make_double2(rin[k], rout[k]) : make_double2(0., 0.);
}

// Four lanes per element (elem_eclipses); lanes past the last element repeat
// it without storing, so that warps stay whole.
__global__ void __launch_bounds__(kThreadsC)
    k_components(__grid_constant__ const CompParams p, ElemRec *el, double4 *pos, DevStatus *st) {
    const int n = p.nd + p.ne + p.ns;
    const int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    const bool in_range = u < n;
    const int i = in_range ? u : n - 1;
    constexpr double EFAC = 1.0000001;
    V3 posn, dirn;
    double area, flux;
    bool trap1 = false;
    if (i < p.nd) {
        // disc: ring k holds elements [off, off + ntheta)
        int lo = 0, hi = p.nrad - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (p.rings[mid].off <= i) lo = mid;
            else hi = mid - 1;
        }
        const DiscRing R = p.rings[lo];
        const int j = i - R.off;
        const double theta = kTwoPi * j / R.ntheta;
        const double sint = sin(theta), cost = cos(theta);
        posn = v3(R.rad * cost, R.rad * sint, R.h);
        dirn = v3(-cost * R.sinp, -sint * R.sinp, R.cosp);
        area = R.area;
        const double r = sqrt(posn.x * posn.x + posn.y * posn.y + posn.z * posn.z);
        flux = p.bright_disc * pow(r / p.rdisc2, p.texp) * (double)(float)area;
    } else if (i < p.nd + p.ne) {
        // outer rim: per longitude, the upper element then NOUT - 1 below it
        const int k = i - p.nd, it = k / p.nout, jj = k % p.nout;
        const double theta = kTwoPi * it / p.ntheta_e;
        const double sint = sin(theta), cost = cos(theta);
        if (jj == 0) {
            posn = v3(EFAC * p.rad_e * cost, EFAC * p.rad_e * sint, EFAC * p.h_e);
            area = p.area_e / 2.;
            trap1 = true;
        } else {
            const int j = jj - 1;
            posn = v3(EFAC * p.rad_e * cost, EFAC * p.rad_e * sint,
                      -p.h_e + 2 * p.h_e * j / (p.nout - 1));
            area = p.area_e;
        }
        dirn = v3(cost, sint, 0);
        // irradiation by the donor as a point source, sunset included
        // (set_disc_continuum.cpp:48-88)
        const V3 vec = v3(1. - posn.x, 0. - posn.y, 0. - posn.z);
        const double r = sqrt(vec.x * vec.x + vec.y * vec.y + vec.z * vec.z);
        const double mu = (dirn.x * vec.x + dirn.y * vec.y + dirn.z * vec.z) / r;
        double temp;
        if (mu >= p.r2) {
            const double geom = sq(p.r2 / r) * mu;
            temp = pow(pow(p.tedge, 4.0) + p.absorb_edge * pow(p.t2, 4.0) * geom, 0.25);
        } else if (mu > -p.r2) {
            const double x0 = -mu / p.r2;
            const double geom = sq(p.r2 / r) * p.r2 *
                                (sqrt(1. - x0 * x0) * (2 + x0 * x0) / 3 - x0 * (kPi / 2 - asin(x0))) /
                                kPi;
            temp = pow(pow(p.tedge, 4.0) + p.absorb_edge * pow(p.t2, 4.0) * geom, 0.25);
        } else {
            temp = p.tedge;
        }
        flux = (double)(float)area * planck(p.wave, temp);
    } else {
        // bright spot: the tilted strip, then the strip parallel to the disc
        const int k = i - p.nd - p.ne, ii = k % p.nspot;
        const bool tilted = k < p.nspot;
        const double dist = p.sfac * ii / (p.nspot - 1);
        const double c = p.length * (dist - p.bmax);
        posn = v3(p.bspot[0] + c * p.bvec[0], p.bspot[1] + c * p.bvec[1], p.bspot[2] + c * p.bvec[2]);
        dirn = tilted ? v3(p.tvec[0], p.tvec[1], p.tvec[2]) : v3(0., 0., 1.);
        area = p.area_s;
        const double bright = p.bright_s * pow(dist / p.bmax, p.expon) *
                              exp(p.expon / p.epow - pow(dist, p.epow));
        flux = bright * (tilted ? (1 - p.cfrac) : p.cfrac) * (double)(float)area;
    }
    ElemRec r;
    r.dx = dirn.x;
    r.dy = dirn.y;
    r.dz = dirn.z;
    r.flux = (float)flux;
    elem_eclipses(p, posn, in_range, p.opaque && i < p.nd + p.ne, trap1, r, st, elem_tag(i));
    if (!in_range || (threadIdx.x & 3) != 0) return;
    el[i] = r;
    pos[i] = make_double4(posn.x, posn.y, posn.z, (double)(float)area);
}

// The disc's ranges of each face, and the partition counts with them: one-range
// and several-range faces per CTA of 256 (k_flat_scatter).
__global__ void __launch_bounds__(256) k_disc_faces(DiscGeom dg, GridDev g, uint8_t *ndx,
                                                    double2 *xr, int32_t *cnt, DevStatus *st) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int ranges = 0;
    if (i < g.n) {
        int nr = 0, s = 0;
        double rin[kDiscRanges], rout[kDiscRanges];
        disc_eclipse(dg, v3(g.px[i], g.py[i], g.pz[i]), nr, rin, rout, kDiscRanges, s);
        if (s) report(st, s, (int)i);
        nr = s ? 0 : (nr < kDiscRanges ? nr : kDiscRanges);
        ndx[i] = (uint8_t)nr;
        for (int k = 0; k < kDiscRanges; k++)
            xr[kDiscRanges * i + k] = k < nr ? make_double2(rin[k], rout[k]) : make_double2(0., 0.);
        ranges = g.necl[i] + nr;
    }
    const int c1 = __syncthreads_count(ranges == 1), c2 = __syncthreads_count(ranges > 1);
    if (threadIdx.x == 0) {
        cnt[blockIdx.x] = c1;
        cnt[gridDim.x + blockIdx.x] = c2;
    }
}

// One CTA per (tile of phase entries, chunk of kElemChunk elements): each
// thread sums the chunk's elements in order for its entry (the chunk staged in
// shared memory, every thread reading the same element: a broadcast) and
// writes three partial sums; k_comp_reduce adds the chunks in order.
constexpr int kElemChunk = 256;

// A range that hides nothing, in the places past an element's last one.
__device__ __forceinline__ double2 no_range() { return make_double2(10., -10.); }

// Elements [t0, t1) of the tile, all of one component, in order. 32 at a time, a lane
// each, their ranges are held against the warp's arc of phases. Where none meets it,
// or hides an element throughout, only mu is tested; elsewhere the first two ranges
// of every element (most have no more), and the rest if some element has them. No
// element branches or votes, so they overlap; one turned away or hidden adds an exact
// zero, as leaving it out does. With a vote and a walk over its ranges per element
// the eclipsed entries' CTAs took 600 cycles an element: 13,800 elements at 2,000
// entries, beside the stars' sweeps, 131 us; 96 so (66 alone).
template <bool LIMB>
__device__ __forceinline__ void comp_run(const ElemRec *tile, int t0, int t1, double ex, double ey,
                                         double ez, double phi, unsigned long long A,
                                         unsigned long long L, double lin, double quad,
                                         double &s) {
    const int lane = threadIdx.x & 31;
    auto value = [&](const ElemRec &r, double mu) {
        const double v = mu * (double)r.flux;  // spot_elem
        if constexpr (!LIMB) return v;
        const double om = 1.0 - mu;
        return v * (1.0 - om * (lin + quad * om));  // disc_elem
    };
    // Point::visible (lcurve.h:81-89)
    auto hides = [&](double2 R) { return (phi >= R.x && phi <= R.y) || phi <= R.y - 1.0; };
    for (int g = t0; g < t1; g += 32) {
        const int end = g + 32 < t1 ? g + 32 : t1;
        int c = kGroupSigns, nr = 0;
        if (g + lane < t1) {
            nr = tile[g + lane].nr;
            c = ranges_class(tile[g + lane].r, nr, A, L);
        }
        if (!__any_sync(0xffffffffu, c != kGroupSigns)) {
#pragma unroll 4
            for (int t = g; t < end; t++) {
                const ElemRec &r = tile[t];
                const double mu = ex * r.dx + ey * r.dy + ez * r.dz;
                const double v = value(r, mu);
                s += mu > 0.0 ? v : 0.0;
            }
            continue;
        }
        if (__all_sync(0xffffffffu, c == kGroupDark || g + lane >= t1)) continue;
        const bool more = __any_sync(0xffffffffu, nr > 2);
#pragma unroll 2
        for (int t = g; t < end; t++) {
            const ElemRec &r = tile[t];
            const double mu = ex * r.dx + ey * r.dy + ez * r.dz;
            bool vis = mu > 0.0 && !hides(r.r[0]) && !hides(r.r[1]);
            if (more)
                for (int k = 2; k < kMaxRanges; k++) vis = vis && !hides(r.r[k]);
            const double v = value(r, mu);
            s += vis ? v : 0.0;
        }
    }
}

__global__ void __launch_bounds__(kThreadsC) k_comp_sums(const ElemRec *__restrict__ el,
                                                         int32_t nd, int32_t ne, int32_t n,
                                                         double lin, double quad, PhaseDev ph,
                                                         double *part, int64_t ldc) {
    __shared__ ElemRec tile[kElemChunk];
    // threads past the last entry repeat it, so that the warp's arc stays narrow
    const int64_t entry = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t e = entry < ph.nent ? entry : ph.nent - 1;
    const double ex = ph.ex[e], ey = ph.ey[e], ez = ph.ez[e], phi = ph.phin[e];
    const unsigned long long pf = ph.pfx[e];
    unsigned long long A, L;
    warp_arc<1>(&pf, A, L);
    const int base = blockIdx.y * kElemChunk;
    const int m = (n - base < kElemChunk) ? n - base : kElemChunk;
    for (int t = threadIdx.x; t < m; t += blockDim.x) {
        ElemRec r = el[base + t];
        r.nr = r.nr < kMaxRanges ? r.nr : kMaxRanges;
#pragma unroll
        for (int k = 0; k < kMaxRanges; k++)
            if (k >= r.nr) r.r[k] = no_range();
        tile[t] = r;
    }
    __syncthreads();
    // the disc's, the rim's and the spot's elements of the chunk
    const int b1 = min(max(nd - base, 0), m), b2 = min(max(nd + ne - base, 0), m);
    double s[3] = {0.0, 0.0, 0.0};
    comp_run<true>(tile, 0, b1, ex, ey, ez, phi, A, L, lin, quad, s[0]);
    comp_run<true>(tile, b1, b2, ex, ey, ez, phi, A, L, lin, quad, s[1]);
    comp_run<false>(tile, b2, m, ex, ey, ez, phi, A, L, lin, quad, s[2]);
    if (entry < ph.nent) {
        double *row = part + 3 * (int64_t)blockIdx.y * ldc;
        row[entry] = s[0];
        row[ldc + entry] = s[1];
        row[2 * ldc + entry] = s[2];
    }
}

__global__ void k_comp_reduce(const double *__restrict__ part, int nchunk, int64_t nent,
                              double *out, int64_t ldc) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nent) return;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int c = 0; c < nchunk; c++) {
        const double *row = part + 3 * (int64_t)c * ldc;
        s0 += row[e];
        s1 += row[ldc + e];
        s2 += row[2 * ldc + e];
    }
    out[e] = s0;
    out[ldc + e] = s1;
    out[2 * ldc + e] = s2;
}

// ---- iscale -------------------------------------------------------------------
// Weighted least squares for the component scale factors, with svdfit's rule
// (svdfit.cpp:22-80): rows of points with sigma z = ferr / sqrt(weight) > 0,
// scaled by 1/z; singular values below 1e-5 of the largest dropped. Here the
// weighted design matrix [A | b] is first reduced by Householder QR (rows of
// points that do not count are zero and change nothing), then R gets a
// one-sided Jacobi SVD (Hestenes 1958): A and R have the same singular values
// and right vectors, so the truncated solution is svdfit's up to rounding.
// One CTA; deterministic tree reductions.
constexpr int kThreadsF = 512;

__device__ double tree_sum(double v, double *sh) {
    const int t = threadIdx.x;
    sh[t] = v;
    __syncthreads();
    for (int w = kThreadsF / 2; w > 0; w >>= 1) {
        if (t < w) sh[t] += sh[t + w];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kThreadsF) k_iscale(int32_t flags, int32_t nc,
                                                      const DatumRec *__restrict__ data, int32_t n,
                                                      const double *__restrict__ fcomp,
                                                      double *work, double *calc, double *sfac,
                                                      double *out) {
    __shared__ double sh[kThreadsF];
    __shared__ double R[6][6], x[5];
    const bool scale = flags & 1, rdata = flags & 2;
    const int t = threadIdx.x;
    if (scale) {
        const int m = nc + 1;  // columns: the components, then b
        double *A = work;      // column-major, n rows
        for (int i = t; i < n; i += kThreadsF) {
            const DatumRec d = data[i];
            const double z = d.weight <= 0. ? -1. : d.ferr / sqrt(d.weight);
            const double invsig = z > 0 ? 1. / z : 0.;
            for (int j = 0; j < nc; j++) A[(int64_t)j * n + i] = invsig * fcomp[5 * (int64_t)i + j];
            A[(int64_t)nc * n + i] = invsig * d.flux;
        }
        __syncthreads();
        for (int j = 0; j < nc; j++) {
            double *cj = A + (int64_t)j * n;
            double p = 0.;
            for (int i = j + t; i < n; i += kThreadsF) p += cj[i] * cj[i];
            const double norm2 = tree_sum(p, sh);
            const double ajj = j < n ? cj[j] : 0.;
            if (norm2 > 0. && j < n) {
                const double alpha = ajj > 0. ? -sqrt(norm2) : sqrt(norm2);
                const double v0 = ajj - alpha;
                const double vnorm2 = norm2 - ajj * ajj + v0 * v0;
                for (int c = j + 1; c < m; c++) {
                    double *cc = A + (int64_t)c * n;
                    double q = t == 0 ? v0 * cc[j] : 0.;
                    for (int i = j + 1 + t; i < n; i += kThreadsF) q += cj[i] * cc[i];
                    const double dot = tree_sum(q, sh);
                    const double f = 2. * dot / vnorm2;
                    if (t == 0) cc[j] -= f * v0;
                    for (int i = j + 1 + t; i < n; i += kThreadsF) cc[i] -= f * cj[i];
                    __syncthreads();
                }
                if (t == 0) cj[j] = alpha;
                __syncthreads();
            }
        }
        if (t == 0) {
            // R (upper nc x nc) and c = (Q^T b)[0 .. nc)
            double c[6];
            for (int i = 0; i < nc; i++) {
                for (int j = 0; j < nc; j++) R[i][j] = (j >= i && i < n) ? A[(int64_t)j * n + i] : 0.;
                c[i] = i < n ? A[(int64_t)nc * n + i] : 0.;
            }
            double V[5][5];
            for (int i = 0; i < nc; i++)
                for (int j = 0; j < nc; j++) V[i][j] = i == j ? 1. : 0.;
            for (int sweep = 0; sweep < 60; sweep++) {
                bool rot = false;
                for (int p = 0; p < nc - 1; p++)
                    for (int q = p + 1; q < nc; q++) {
                        double al = 0., be = 0., ga = 0.;
                        for (int i = 0; i < nc; i++) {
                            al += R[i][p] * R[i][p];
                            be += R[i][q] * R[i][q];
                            ga += R[i][p] * R[i][q];
                        }
                        if (ga == 0. || fabs(ga) <= 1e-15 * sqrt(al * be)) continue;
                        rot = true;
                        const double zeta = (be - al) / (2. * ga);
                        const double tt = (zeta >= 0. ? 1. : -1.) / (fabs(zeta) + sqrt(1. + zeta * zeta));
                        const double cs = 1. / sqrt(1. + tt * tt), sn = cs * tt;
                        for (int i = 0; i < nc; i++) {
                            const double ap = R[i][p], aq = R[i][q];
                            R[i][p] = cs * ap - sn * aq;
                            R[i][q] = sn * ap + cs * aq;
                            const double vp = V[i][p], vq = V[i][q];
                            V[i][p] = cs * vp - sn * vq;
                            V[i][q] = sn * vp + cs * vq;
                        }
                    }
                if (!rot) break;
            }
            double w[5], wmax = 0.;
            for (int j = 0; j < nc; j++) {
                double s2 = 0.;
                for (int i = 0; i < nc; i++) s2 += R[i][j] * R[i][j];
                w[j] = sqrt(s2);
                wmax = fmax(wmax, w[j]);
            }
            for (int k = 0; k < 5; k++) x[k] = 0.;
            for (int j = 0; j < nc; j++) {
                if (!(w[j] >= 1e-5 * wmax) || w[j] == 0.) continue;
                double ub = 0.;
                for (int i = 0; i < nc; i++) ub += R[i][j] * c[i];
                ub /= w[j] * w[j];
                for (int k = 0; k < nc; k++) x[k] += V[k][j] * ub;
            }
            for (int k = 0; k < 5; k++) sfac[k] = k < nc ? x[k] : 0.;
        }
        __syncthreads();
    }
    // calc from the components (light_curve_comp.cpp:532-556)
    double cs = 0., ws = 0.;
    const double s0 = sfac[0], s1 = sfac[1], s2 = sfac[2], s3 = sfac[3], s4 = sfac[4];
    for (int i = t; i < n; i += kThreadsF) {
        const double *f = fcomp + 5 * (int64_t)i;
        double c = s0 * f[0] + s1 * f[1] + s2 * f[2] + s3 * f[3];
        if (nc == 5) c += s4 * f[4];
        calc[i] = c;
        const DatumRec d = data[i];
        if (d.weight > 0.) {
            ws += d.weight;
            cs += d.weight * sq((d.flux - c) / d.ferr);
        }
    }
    const double chisq = tree_sum(cs, sh), wnok = tree_sum(ws, sh);
    if (t == 0 && (scale || rdata)) {
        out[0] = chisq;
        out[1] = wnok;
        out[2] = 1.;
    } else if (t == 0) {
        out[2] = 0.;
    }
}

int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_components(const CompParams &p, ElemRec *el, double4 *pos, DevStatus *st,
                       cudaStream_t s) {
    const int n = p.nd + p.ne + p.ns;
    if (n <= 0) return;
    k_components<<<nblk(4 * (int64_t)n, kThreadsC), kThreadsC, 0, s>>>(p, el, pos, st);
    count_launch();
}

void launch_disc_faces(const DiscGeom &dg, const GridDev &g, uint8_t *ndx, double2 *xr,
                       int32_t *cnt, DevStatus *st, cudaStream_t s) {
    if (g.n <= 0) return;
    k_disc_faces<<<nblk(g.n, 256), 256, 0, s>>>(dg, g, ndx, xr, cnt, st);
    count_launch();
}

int64_t comp_sums_scratch(int32_t n, int64_t ldc) {
    return 3 * (int64_t)((n + kElemChunk - 1) / kElemChunk) * ldc;
}

void launch_comp_sums(const ElemRec *el, int32_t nd, int32_t ne, int32_t n, double lin,
                      double quad, const PhaseDev &ph, double *part, double *out, int64_t ldc,
                      cudaStream_t s) {
    if (ph.nent <= 0) return;
    const int nchunk = (n + kElemChunk - 1) / kElemChunk;
    if (nchunk == 0) {
        cudaMemsetAsync(out, 0, 3 * ldc * sizeof(double), s);
        return;
    }
    k_comp_sums<<<dim3(nblk(ph.nent, kThreadsC), nchunk), kThreadsC, 0, s>>>(el, nd, ne, n, lin,
                                                                             quad, ph, part, ldc);
    count_launch();
    k_comp_reduce<<<nblk(ph.nent, 256), 256, 0, s>>>(part, nchunk, ph.nent, out, ldc);
    count_launch();
}

void launch_iscale(int32_t flags, int32_t nc, const DatumRec *data, int32_t n,
                   const double *fcomp, double *work, double *calc, double *sfac, double *out,
                   cudaStream_t s) {
    k_iscale<<<1, kThreadsF, 0, s>>>(flags, nc, data, n, fcomp, work, calc, sfac, out);
    count_launch();
}

// ---- host setup -------------------------------------------------------------

namespace eng {

namespace {

// The gas stream's motion (rocacc.cpp: the restricted three-body problem in the
// rotating frame, in the orbital plane, where the stream starts at rest in z)
// by Taylor series (e.g. Jorba & Zou 2005): with p_i = r_i^-3 the equations
//   x'' =  2 y' + x - f2 - f1 p1 x - f2 p2 (x - 1)
//   y'' = -2 x' + y - f1 p1 y - f2 p2 y
// give the next coefficients of x and y from the lower ones, those of p_i
// following from r_i^2 by the recurrence of a power. Order kOrder with steps at
// which the last terms are 1e-16 of the coordinates: some 20 steps, where a
// fifth-order Runge-Kutta pair at 1e-13 took 5000.
constexpr int kOrder = 26;
struct StreamSeries {
    double x[kOrder + 1], y[kOrder + 1];

    void expand(double q, const double *s) {  // s = x, y, x', y'
        const double f1 = 1. / (1. + q), f2 = f1 * q;
        double s1[kOrder], s2[kOrder], p1[kOrder], p2[kOrder];
        x[0] = s[0]; x[1] = s[2];
        y[0] = s[1]; y[1] = s[3];
        for (int n = 0; n + 2 <= kOrder; n++) {
            // r^2 about either star (x - 1 differs from x in its first coefficient)
            double xx = 0., yy = 0.;
            for (int k = 0; k <= n; k++) {
                xx += x[k] * x[n - k];
                yy += y[k] * y[n - k];
            }
            s1[n] = xx + yy;
            s2[n] = s1[n] - 2. * x[n] + (n == 0 ? 1. : 0.);
            if (n == 0) {
                p1[0] = 1. / (s1[0] * sqrt(s1[0]));
                p2[0] = 1. / (s2[0] * sqrt(s2[0]));
            } else {
                double a1 = 0., a2 = 0.;
                for (int k = 0; k < n; k++) {
                    const double c = -1.5 * (n - k) - k;
                    a1 += c * s1[n - k] * p1[k];
                    a2 += c * s2[n - k] * p2[k];
                }
                p1[n] = a1 / (n * s1[0]);
                p2[n] = a2 / (n * s2[0]);
            }
            double px1 = 0., px2 = 0., py = 0.;
            for (int k = 0; k <= n; k++) {
                px1 += p1[k] * x[n - k];
                px2 += p2[k] * x[n - k];
                py += (f1 * p1[k] + f2 * p2[k]) * y[n - k];
            }
            px2 -= p2[n];
            const double d = (n + 1.) * (n + 2.);
            x[n + 2] = (2. * (n + 1) * y[n + 1] + x[n] - (n == 0 ? f2 : 0.) - f1 * px1 - f2 * px2) / d;
            y[n + 2] = (-2. * (n + 1) * x[n + 1] + y[n] - py) / d;
        }
    }
    // the step whose last two terms stay below 1e-16 of the start's coordinates
    double step() const {
        const double scale = 1e-16 * std::max(fabs(x[0]), fabs(y[0]));
        double h = 1.;
        for (int n = kOrder - 1; n <= kOrder; n++) {
            const double c = std::max(fabs(x[n]), fabs(y[n]));
            if (c > 0.) h = std::min(h, pow(scale / c, 1. / n));
        }
        return h;
    }
    void at(double t, double *s) const {
        double a = 0., b = 0., da = 0., db = 0.;
        for (int n = kOrder; n >= 1; n--) {
            da = da * t + n * x[n];
            db = db * t + n * y[n];
            a = (a + x[n]) * t;
            b = (b + y[n]) * t;
        }
        s[0] = a + x[0];
        s[1] = b + y[0];
        s[2] = da;
        s[3] = db;
    }
};

double radius(const double *s) { return sqrt(sq(s[0]) + sq(s[1])); }
double outward(const double *s) { return s[0] * s[2] + s[1] * s[3]; }  // r dr/dt

}  // namespace

// Where the gas stream from L1 first reaches distance rad from star 1:
// Roche::strinit's start (strining.cpp:14-33) and the motion of rocacc.cpp,
// integrated by Taylor series, the crossing bisected in time to the last bits.
// The reference integrates with a Bulirsch-Stoer stepper whose first step size
// is kept in a static between calls (stradv.cpp:35), to 1e-10 in radius, so the
// two agree to its error, not bit for bit.
bool bright_spot_position(double q, double rad, double *pos, Fail &f) {
    const double SMALL = 1.e-5, TMAX = 10.;
    const double rl1 = xl1(q);
    if (rl1 < 0) {
        f = {LCG_E_NOCONVERGE, "Roche::xl1(double): exceeded maximum iterations"};
        return false;
    }
    const double mu = q / (1.0 + q);
    const double a = (1.0 - mu) / pow(rl1, 3) + mu / pow((1. - rl1), 3);
    const double lambda1 = sqrt(((a - 2.0) + sqrt(a * (9.0 * a - 8.0))) / 2.0);
    const double m1 = (lambda1 * lambda1 - 2.0 * a - 1.0) / 2.0 / lambda1;
    double s[4] = {rl1 - SMALL, -m1 * SMALL, -lambda1 * SMALL, -lambda1 * m1 * SMALL};
    const double rinit = radius(s);
    auto before = [&](double r) { return (rinit > rad && r > rad) || (rinit < rad && r < rad); };
    double t = 0.;
    for (int guard = 0; before(radius(s)); guard++) {
        if (guard > 100000 || t > TMAX) {
            f = {LCG_E_ROCHE, "Roche::stradv: taken too long without crossing radius"};
            return false;
        }
        StreamSeries S;
        S.expand(q, s);
        const double h = S.step();
        // the radius within the step: at 16 times, and at a turning point between
        // two of them, where it may cross and come back
        double lo = 0., slo[4] = {s[0], s[1], s[2], s[3]}, shi[4];
        bool crossed = false;
        for (int k = 1; k <= 16 && !crossed; k++) {
            double hi = h * k / 16;
            S.at(hi, shi);
            if (before(radius(shi)) && (outward(slo) > 0.) != (outward(shi) > 0.)) {
                double ta = lo, tb = hi, sm[4];
                const bool up = outward(slo) > 0.;
                for (int i = 0; i < 60; i++) {
                    const double tm = (ta + tb) / 2.;
                    S.at(tm, sm);
                    if ((outward(sm) > 0.) == up) ta = tm;
                    else tb = tm;
                }
                if (!before(radius(sm))) {
                    hi = (ta + tb) / 2.;
                    S.at(hi, shi);
                }
            }
            if (!before(radius(shi))) {
                for (int i = 0; i < 60; i++) {
                    const double tm = (lo + hi) / 2.;
                    double sm[4];
                    S.at(tm, sm);
                    if (before(radius(sm))) lo = tm;
                    else hi = tm;
                }
                S.at(hi, shi);
                crossed = true;
            }
            lo = hi;
            std::copy(shi, shi + 4, slo);
        }
        std::copy(slo, slo + 4, s);
        t += h;
        if (crossed) break;
    }
    pos[0] = s[0];
    pos[1] = s[1];
    pos[2] = 0.;
    return true;
}

// Lobe checks and reference spheres of set_disc_grid / set_disc_edge /
// set_bright_spot_grid (set_disc_grid.cpp:31-66), with the reference's
// message for the component that raises it.
static bool comp_radii(const lcg_model &m, const char *who, CompParams &p, double &rdisc1,
                       Fail &f) {
    double r1, r2;
    get_r1r2(m, r1, r2);
    const double rl1 = xl11(m.q, m.spin1), rl2 = 1. - xl12(m.q, m.spin2);
    char b[160];
    if (r1 < 0) r1 = rl1;
    else if (r1 > rl1) {
        snprintf(b, sizeof b, "%s: the primary star is larger than its Roche lobe!", who);
        f = {LCG_E_LOBE, b};
        return false;
    }
    if (r2 < 0) r2 = rl2;
    else if (r2 > rl2) {
        snprintf(b, sizeof b, "%s: the secondary star is larger than its Roche lobe!", who);
        f = {LCG_E_LOBE, b};
        return false;
    }
    p.r1 = r1;
    p.r2 = r2;
    p.spin1 = m.spin1;
    p.spin2 = m.spin2;
    ref_sphere(kStar1, m.q, m.spin1, r1 / rl1, p.rref1, p.pref1);
    ref_sphere(kStar2, m.q, m.spin2, r2 / rl2, p.rref2, p.pref2);
    rdisc1 = m.rdisc1 > 0. ? m.rdisc1 : r1;
    return true;
}

bool comp_setup(const lcg_model &m, CompParams &p, std::vector<DiscRing> &rings, Fail &f) {
    p = CompParams{};
    rings.clear();
    const double ri = deg2rad(m.iangle);
    p.q = m.q;
    p.cosi = cos(ri);
    p.sini = sin(ri);
    p.delta = m.delta_phase;
    p.eclipse1 = m.eclipse1;
    p.eclipse2 = m.eclipse2;
    p.roche1 = m.roche1;
    p.roche2 = m.roche2;
    p.wave = m.wavelength;
    const double rdisc2 = m.rdisc2 > 0. ? m.rdisc2 : m.radius_spot;
    double rdisc1 = 0.;
    if (m.add_disc) {
        if (!comp_radii(m, "set_disc_grid", p, rdisc1, f)) return false;
        const double EFAC = 1.0000001;
        const double drad = (rdisc2 - rdisc1) / m.nrad, drrad = rdisc2 / m.nrad;
        int off = 0;
        for (int i = 0; i < m.nrad; i++) {
            DiscRing R;
            R.rad = rdisc1 + (rdisc2 - rdisc1) * (i + 0.5) / m.nrad;
            int nt = int(ceil(kTwoPi * R.rad / drrad));
            R.ntheta = nt > 8 ? nt : 8;
            R.h = EFAC * m.height_disc * pow(R.rad, m.beta_disc);
            const double tanp = m.beta_disc * R.h / R.rad;
            R.cosp = 1. / sqrt(1 + sq(tanp));
            R.sinp = tanp * R.cosp;
            R.area = kTwoPi / R.ntheta * R.rad * drad;
            R.off = off;
            off += R.ntheta;
            rings.push_back(R);
        }
        p.nd = off;
        p.nrad = m.nrad;
        p.bright_disc = planck(m.wavelength, m.temp_disc);
        p.rdisc2 = rdisc2;
        p.texp = m.texp_disc;
        // the outer rim (set_disc_edge with outer = true)
        const double size = rdisc2 / m.nrad;
        p.rad_e = rdisc2;
        p.h_e = m.height_disc * pow(p.rad_e, m.beta_disc);
        p.nout = int(2 * p.h_e / size) + 2;
        const int nt = int(ceil(kTwoPi * p.rad_e / size));
        p.ntheta_e = nt > 8 ? nt : 8;
        p.area_e = kTwoPi / p.ntheta_e * p.rad_e * 2 * p.h_e / (p.nout - 1);
        p.ne = p.ntheta_e * p.nout;
        p.tedge = m.temp_edge;
        p.t2 = fabs(m.t2);
        p.absorb_edge = m.absorb_edge;
        p.opaque = m.opaque;
        if (m.opaque && m.beta_disc < 1 && (p.nd + p.ne) > 0) {
            f = {LCG_E_ROCHE, "Roche::disc_eclipse: beta must be >= 1"};
            return false;
        }
    }
    p.dg = DiscGeom{sin(kPi / 180. * m.iangle), cos(kPi / 180. * m.iangle), rdisc1, rdisc2,
                    m.beta_disc, m.height_disc};
    if (m.add_spot) {
        double rd1;
        if (!comp_radii(m, "set_bright_spot_grid", p, rd1, f)) return false;
        if (m.nspot < 2) {
            f = {LCG_E_INVALID, "set_bright_spot_grid: nspot must be at least 2"};
            return false;
        }
        if (!bright_spot_position(m.q, m.radius_spot, p.bspot, f)) return false;
        const double theta =
            atan2(p.bspot[1], p.bspot[0]) + kTwoPi / 4. + deg2rad(m.angle_spot);
        const double alpha = deg2rad(m.yaw_spot), tilt = deg2rad(m.tilt_spot);
        p.bvec[0] = cos(theta); p.bvec[1] = sin(theta); p.bvec[2] = 0;
        p.tvec[0] = sin(tilt) * sin(theta + alpha);
        p.tvec[1] = -sin(tilt) * cos(theta + alpha);
        p.tvec[2] = cos(tilt);
        p.bmax = pow(m.expon_spot / m.epow_spot, 1. / m.epow_spot);
        p.sfac = 20. + p.bmax;
        p.area_s = p.sfac * m.length_spot * m.height_spot / (m.nspot - 1);
        p.bright_s = planck(m.wavelength, m.temp_spot);
        p.expon = m.expon_spot;
        p.epow = m.epow_spot;
        p.cfrac = m.cfrac_spot;
        p.length = m.length_spot;
        p.nspot = m.nspot;
        p.ns = 2 * m.nspot;
    }
    for (int star = 0; star < 2; star++) {
        EclParams &e = p.ecl[star];
        const bool one = star == kStar1;
        e.comp_star = star;
        e.comp_roche = one ? p.roche1 : p.roche2;
        e.q = p.q;
        e.comp_spin = one ? p.spin1 : p.spin2;
        e.comp_rref = one ? p.rref1 : p.rref2;
        e.comp_pref = one ? p.pref1 : p.pref2;
        e.comp_r = one ? p.r1 : p.r2;
        e.cosi = p.cosi;
        e.sini = p.sini;
        e.delta = p.delta;
        e.edge = make_edge_star(star, e.q, e.comp_spin, e.cosi, e.sini, e.comp_rref, e.comp_pref);
    }
    return true;
}

}  // namespace eng
}  // namespace lcg
