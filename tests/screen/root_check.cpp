// Host check of the eclipse boundaries found from their roots
// (lcurve_re_b200/csrc/ecl_root.cuh) against the bisection with Roche::fblink.
//
// The device code (eclipse.cuh, ecl_root.cuh) is compiled here for the host,
// with the CUDA qualifiers defined away. For every face of the grid given on
// stdin (as screen_check.cpp takes it; a negative radius fills the lobe) it
// runs the sphere test and pot_min, then walks both bisections with fblink
// and compares what edge_zone's intervals, eval_edge and fblink_edge say of
// every midpoint, and of phases drawn inside the intervals and just beyond
// their ends. Prints "hits tests by_zone evaluations searches wrong" and
// exits 1 if any answer differs from fblink's.
#include <cstdio>
#include <cstdlib>
#include <vector>
#define __device__
#define __noinline__
#define __forceinline__ inline
static struct { unsigned x; } threadIdx;
#define __shfl_sync(m, v, l) (v)
#define __shfl_xor_sync(m, v, l) (v)
#define __any_sync(m, p) (p)
#define __ballot_sync(m, p) ((p) ? 1u : 0u)
#define __clz(x) __builtin_clz(x)
#include "../../lcurve_re_b200/csrc/eclipse.cuh"
#include "../../lcurve_re_b200/csrc/ecl_root.cuh"
using namespace lcg;

int main() {
    double h[8];
    long long n = 0;
    if (fread(h, 8, 8, stdin) != 8 || fread(&n, 8, 1, stdin) != 1) return 2;
    std::vector<double> pos(3 * (size_t)n);
    if (fread(pos.data(), 8, pos.size(), stdin) != pos.size()) return 2;
    const double q = h[0], cosi = h[1], sini = h[2], delta = h[3], spin = h[4];
    const int star = (int)h[7];
    const double rl = star == kStar1 ? xl11(q, spin) : 1. - xl12(q, spin);
    const double rad = h[5] < 0. ? rl : h[5];
    double rref, pref;
    ref_sphere(star, q, spin, rad / rl, rref, pref);
    const EdgeStar S = make_edge_star(star, q, spin, cosi, sini, rref, pref);
    const V3 cofm = star == kStar1 ? v3(0., 0., 0.) : v3(1., 0., 0.);
    long long hits = 0, tests = 0, zone = 0, evals = 0, searches = 0, wrong = 0;
    for (long long i = 0; i < n; i++) {
        const V3 r = v3(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]);
        double phi1, phi2, lam1, lam2, phi, lam;
        if (!sphere_eclipse_ph(cosi, sini, r, cofm, rref, phi1, phi2, lam1, lam2)) continue;
        const double acc = 2. * sqrt(2. * kTwoPi * (lam2 - lam1) * delta);
        int st = 0;
        if (!pot_min(star, q, spin, cosi, sini, r, phi1, phi2, lam1, lam2, rref, pref, acc, phi,
                     lam, st))
            continue;
        hits++;
        const V3 u0 = sub(r, cofm);
        const double u2 = norm2(u0);
        auto truth = [&](double ph) {
            return fblink(star, q, spin, acc, set_earth(cosi, sini, ph), r, rref, pref, st)
                       ? kEdgeTrue
                       : kEdgeFalse;
        };
        for (int side = 0; side < 2; side++) {
            double pin = phi, pout = side ? phi2 : phi1;
            const double dir = pout > pin ? 1. : -1.;
            const EdgeZone z = edge_zone(S, u0, acc, delta, pin, pout);
            while (fabs(pin - pout) > delta) {
                const double pmid = (pin + pout) / 2.;
                const int is = truth(pmid);
                const int said[3] = {zone_test(z, dir, pmid),
                                     eval_edge(S, u0, u2, acc, pmid, 0.).ans,
                                     fblink_edge(S, u0, u2, acc, pmid)};
                for (int a : said) wrong += a != kEdgeUnsure && a != is;
                tests++;
                if (said[0] != kEdgeUnsure) zone++;
                else if (!zone_between(z, dir, pmid) && said[1] != kEdgeUnsure) evals++;
                else searches++;
                if (is == kEdgeTrue) pin = pmid;
                else pout = pmid;
            }
            for (int k = 0; k < 6; k++) {  // within the intervals, dense at their inner ends
                const double w = (double)rand() / RAND_MAX, w4 = w * w * w * w;
                const double ph[2] = {z.hc + dir * (z.hid - w4 * (z.hrad + z.hid)),
                                      z.vc + dir * (z.vis + w4 * (z.vrad - z.vis))};
                for (double p : ph) {
                    const int a = zone_test(z, dir, p);
                    wrong += a != kEdgeUnsure && a != truth(p);
                }
                const double at[2] = {z.hc + dir * (z.hid - 30. * delta * w4),
                                      z.vc + dir * (z.vis + 30. * delta * w4)};
                for (double p : at) {
                    const int a = zone_test(z, dir, p);
                    wrong += a != kEdgeUnsure && a != truth(p);
                }
            }
        }
    }
    printf("%lld %lld %lld %lld %lld %lld\n", hits, tests, zone, evals, searches, wrong);
    return wrong ? 1 : 0;
}
