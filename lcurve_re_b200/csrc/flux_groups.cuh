// flux_groups.cuh — what a warp of a flux sweep can tell about a group of faces
// from its record (RunRec, engine.h) and its own entries; shared by the mixed
// and the FP64 sweeps.
#pragma once

#include "engine.h"
#include "fixed_phase.cuh"

namespace lcg {
namespace {

// The warp's phase arc: every entry of the warp lies in [A, A + L] (mod 2^64),
// A its first lane's first entry. For time-ordered points it is a short arc of
// the orbit; in any order it still holds every entry.
template <int PPT>
__device__ __forceinline__ void warp_arc(const unsigned long long *pf, unsigned long long &A,
                                         unsigned long long &L) {
    A = __shfl_sync(0xffffffffu, pf[0], 0);
    unsigned long long l = 0ull;
#pragma unroll
    for (int j = 0; j < PPT; j++) {
        const unsigned long long d = pf[j] - A;
        if (d > l) l = d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, l, o);
        l = t > l ? t : l;
    }
    L = l;
}

// What the warp knows of a group of faces: which of its entries could see it
// and whether a range could hide it (warp-uniform).
enum { kGroupDark = 0, kGroupBright = 1, kGroupSigns = 2, kGroupRanges = 3 };

// The arc [A, A + L] of the warp's phases against a group's ranges, exact on the
// circle: all faces hidden throughout it, some range meeting it, or none.
__device__ __forceinline__ int arc_class(const RunRec &R, unsigned long long A,
                                         unsigned long long L) {
    const ulonglong2 H = R.hull;
    if (!(H.y == ~0ull || (H.y != 0ull && ((H.x - A) <= L || (A - H.x) < H.y))))
        return kGroupSigns;
    const unsigned long long o = A - R.all.x;
    return o < R.all.y && L < R.all.y - o ? kGroupDark : kGroupRanges;
}

// One range [in, out], as the double-precision sweeps test it, against the arc: hidden
// throughout (kGroupDark), met (kGroupRanges) or not (kGroupSigns). Its ends are drawn
// in or out by two units; a range that a turn does not hold as it is counts as met.
__device__ __forceinline__ int range_class(double in, double out, unsigned long long A,
                                           unsigned long long L) {
    if (!(in >= 0. && in < 1. && out >= in)) return kGroupRanges;
    if (out - 1.0 >= in) return kGroupDark;
    const ulonglong2 E = ecl_fx64(in, out);
    if (E.y >= ~0ull - 4ull) return kGroupRanges;
    const unsigned long long x = E.x - 2ull;
    if (x - A > L && A - x >= E.y + 4ull) return kGroupSigns;
    const unsigned long long o = A - (E.x + 2ull), y = E.y > 4ull ? E.y - 4ull : 0ull;
    return o < y && L < y - o ? kGroupDark : kGroupRanges;
}

// An element's ranges together.
__device__ __forceinline__ int ranges_class(const double2 *r, int nr, unsigned long long A,
                                            unsigned long long L) {
    int c = kGroupSigns;
    for (int k = 0; k < nr; k++) {
        const int q = range_class(r[k].x, r[k].y, A, L);
        if (q == kGroupDark) return q;
        if (q == kGroupRanges) c = q;
    }
    return c;
}

}  // namespace
}  // namespace lcg
