// Host check of the surface radii found from their roots (face_chop_root,
// lcurve_re_b200/csrc/ecl_root.cuh) against face_chop's plain walk. Arguments:
// q spin radius(<0: fills the lobe) star acc ndir. Directions cover the sphere
// and crowd around the line of centres. Prints "directions differ" and exits 1
// if any radius or failure code differs.
#include <cstdio>
#include <cstdlib>
#include "../../lcurve_re_b200/csrc/ecl_root.cuh"
using namespace lcg;

int main(int argc, char **argv) {
    if (argc < 7) return 2;
    const double q = atof(argv[1]), spin = atof(argv[2]);
    const int star = atoi(argv[4]);
    const double acc = atof(argv[5]);
    const int nd = atoi(argv[6]);
    const double rl = star == kStar1 ? xl11(q, spin) : 1. - xl12(q, spin);
    const double rad = atof(argv[3]) < 0. ? rl : atof(argv[3]);
    double rref, pref;
    ref_sphere(star, q, spin, rad / rl, rref, pref);
    const EdgeStar S = make_edge_star(star, q, spin, 0., 0., rref, pref);
    long long n = 0, bad = 0;
    for (int i = 0; i < nd; i++)
        for (int j = 0; j < 24; j++) {
            // cosine of the angle from the axis: uniform, and crowding at both ends
            const double u = (i + 0.5) / nd;
            const double c = (i & 3) == 0   ? 1. - u * u * u * u
                             : (i & 3) == 1 ? -1. + u * u * u * u
                                            : 2. * u - 1.;
            const double s = sqrt(1. - c * c), a = kTwoPi * (j + 0.3) / 24;
            double r0 = 0., r1 = 0.;
            const int f0 = face_chop(star, q, spin, c, s * cos(a), rref, pref, acc, r0);
            const int f1 = face_chop_root(S, star, q, spin, c, s * cos(a), rref, pref, acc, r1);
            n++;
            bad += f0 != f1 || r0 != r1;
        }
    for (int k = -1; k <= 1; k += 2) {  // the line of centres itself
        double r0 = 0., r1 = 0.;
        const int f0 = face_chop(star, q, spin, k, 0., rref, pref, acc, r0);
        const int f1 = face_chop_root(S, star, q, spin, k, 0., rref, pref, acc, r1);
        n++;
        bad += f0 != f1 || r0 != r1;
    }
    printf("%lld %lld\n", n, bad);
    return bad ? 1 : 0;
}
