// flux64.cu — FP64 multi-phase flux sweep with the reference's arithmetic.
//
// Same sums as sum_star{1,2}_multi_t (comp_light_flat.cpp:241-372): faces in
// blocks of 1024 (FACE_BLOCK, :239) in FlatGrid order; per block and phase
// entry, element values of s1_elem / s2_elem (:109-168) are added in
// ascending face order; k_reduce_chunks then adds the block partials in block
// order. Compiled with --fmad=false, every operation rounds as in the
// reference, so given the same FlatGrid and phases the result is
// bit-identical (sqrt and division are IEEE on both sides).
//
// A CTA owns one 1024-face block and a tile of phase entries; the block's
// SoA columns are staged into shared memory by bulk TMA copies.
#include "engine.h"
#include "flux_groups.cuh"
#include "tma.cuh"

namespace lcg {

namespace {

constexpr int kThreads64 = 256;
constexpr int kThreadsRag = 128;  // several-range faces
constexpr int kBlock = 1024;

struct Consts64 {
    double c1, c2, c3, c4, base, mucrit, beam, spin, vfac, xcofm, rlens1;
};

// imu_bl (comp_light_flat.cpp:80-95)
template <int LT>
__device__ __forceinline__ double imu_bl(double mu, const Consts64 &L) {
    const double m = (1.0 < mu) ? 1.0 : mu;
    double im;
    if constexpr (LT == 0) {
        const double om = 1.0 - m;
        im = 1.0 - om * (L.c1 + om * (L.c2 + om * (L.c3 + om * L.c4)));
    } else {
        const double msq = sqrt((m < 0.0) ? 0.0 : m);
        im = L.base + msq * (L.c1 + msq * (L.c2 + msq * (L.c3 + msq * L.c4)));
    }
    return (double)(mu > 0.0) * im;
}

// mu = e . n, in the reference's order of operations
__device__ __forceinline__ double mu_of(double ex, double ey, double ez, double dx, double dy,
                                        double dz) {
    return ex * dx + ey * dy + ez * dz;
}

// Elements at or below this mu are exactly zero: the factor (mu > mucrit)
// and, without beaming, (mu > 0) inside imu_bl multiply a finite value.
template <bool BEAM>
__device__ __forceinline__ double zero_below(const Consts64 &L) {
    return BEAM ? L.mucrit : (L.mucrit > 0.0 ? L.mucrit : 0.0);
}

// s1_elem / s2_elem (comp_light_flat.cpp:109-168), given mu
template <int LT, bool BEAM, bool GLENS, int STAR>
__device__ __forceinline__ double elem_mu(double mu, double ex, double ey, double ez, double dx,
                                          double dy, double px, double py, double pz,
                                          double flux, const Consts64 &L) {
    double magn = 1.0;
    if constexpr (GLENS) {
        const double d = -(px * ex + py * ey + pz * ez);
        const double qx = px + d * ex, qy = py + d * ey, qz = pz + d * ez;
        const double p = sqrt(qx * qx + qy * qy + qz * qz);
        const double ph = 0.5 * p;
        const double rd = L.rlens1 * d;
        const double pd = (ph * ph > 25.0 * rd) ? p + rd / p : ph + sqrt(ph * ph + rd);
        const double mg = pd * pd / (pd - ph) / ph / 4.0;
        magn = d > 0.0 ? mg : 1.0;
    }
    double val;
    if constexpr (!BEAM) {
        if constexpr (STAR == 0) val = mu * flux * imu_bl<LT>(mu, L);
        else val = mu * magn * flux * imu_bl<LT>(mu, L);
    } else {
        const double vx = -L.vfac * L.spin * py;
        const double vy = STAR == 0 ? L.vfac * (L.spin * px - L.xcofm)
                                    : L.vfac * (L.spin * (px - 1.0) + 1.0 - L.xcofm);
        const double vr = -(ex * vx + ey * vy);
        const double vn = dx * vx + dy * vy;
        const double mud = mu - mu * vr - vn;
        if constexpr (STAR == 0) val = mu * flux * (1.0 - L.beam * vr) * imu_bl<LT>(mud, L);
        else val = mu * magn * flux * (1.0 - L.beam * vr) * imu_bl<LT>(mud, L);
    }
    if constexpr (GLENS) return mu > L.mucrit ? val : 0.0;
    return (double)(mu > L.mucrit) * val;
}

// A thread's entry, in FP32 for the group tests: earth vector, the length of its
// xy part, and the phase arc of its warp.
struct Arc64 {
    float ex, ey, ez, exy;
    unsigned long long A, L;
};

// What a group of faces is to a warp's entries (flux_groups.cuh): dark when mu is
// at or below zb, or every face eclipsed, at all of them; bright when mu lies
// above zb for every face and entry and no range reaches the warp's arc. The
// bounds are FP32; 2e-6 covers the rounding for vectors of length one. Longer
// ones and NaN come as NaN, which is neither dark nor bright.
template <bool ECL>
__device__ __forceinline__ int group64(const RunRec &R, float zb, const Arc64 &W) {
    const float d = W.ex * R.ax + W.ey * R.ay, q = W.exy * R.r;
    const float z0 = W.ez * R.cmin, z1 = W.ez * R.cmax;
    if (!__any_sync(0xffffffffu, !(q + d + fmaxf(z0, z1) + 2e-6f < zb))) return kGroupDark;
    if constexpr (ECL) {
        const int c = arc_class(R, W.A, W.L);
        if (c != kGroupSigns) return c;
    }
    return __all_sync(0xffffffffu, d - q + fminf(z0, z1) - 2e-6f > zb) ? kGroupBright
                                                                       : kGroupSigns;
}

struct Cols64 {  // a staged block's columns
    const double *dx, *dy, *dz, *fl, *in, *out, *px, *py, *pz;
};

struct Entry64 {
    double ex, ey, ez, pn;
};

// Faces [t0, t1) of the block, every one visible at every entry (no beaming, no
// lensing): s1_elem / s2_elem without the factors that are one there, (mu > 0)
// and (mu > mucrit).
template <int LT>
__device__ __forceinline__ void bright64(const Cols64 &C, int t0, int t1, const Entry64 &E,
                                         const Consts64 &L, double &br) {
#pragma unroll 4
    for (int t = t0; t < t1; t++) {
        const double mu = mu_of(E.ex, E.ey, E.ez, C.dx[t], C.dy[t], C.dz[t]);
        const double m = (1.0 < mu) ? 1.0 : mu;
        double im;
        if constexpr (LT == 0) {
            const double om = 1.0 - m;
            im = 1.0 - om * (L.c1 + om * (L.c2 + om * (L.c3 + om * L.c4)));
        } else {
            const double msq = sqrt(m);
            im = L.base + msq * (L.c1 + msq * (L.c2 + msq * (L.c3 + msq * L.c4)));
        }
        br += mu * C.fl[t] * im;
    }
}

// The same faces with every factor, and the range when ECL. Per face, one vote
// of the warp: at or below zb (exactly zero) or eclipsed at every entry of the
// warp, its elements would add exact zeros, and the warp moves on.
template <int LT, bool BEAM, bool GLENS, int STAR, bool ECL>
__device__ __forceinline__ void faces64(const Cols64 &C, int t0, int t1, const Entry64 &E,
                                        double zb, const Consts64 &L, double &br) {
    constexpr bool need_pos = BEAM || GLENS;
#pragma unroll 1
    for (int t = t0; t < t1; t++) {
        const double dx = C.dx[t], dy = C.dy[t], dz = C.dz[t];
        double ein = 0., eout = 0.;
        if constexpr (ECL) { ein = C.in[t]; eout = C.out[t]; }
        const double mu = mu_of(E.ex, E.ey, E.ez, dx, dy, dz);
        const bool ecl = ECL && ((E.pn >= ein && E.pn <= eout) || E.pn <= eout - 1.0);
        if (!__any_sync(0xffffffffu, (mu > zb) && !ecl)) continue;
        double px = 0., py = 0., pz = 0.;
        if constexpr (need_pos) { px = C.px[t]; py = C.py[t]; pz = C.pz[t]; }
        const double v = elem_mu<LT, BEAM, GLENS, STAR>(mu, E.ex, E.ey, E.ez, dx, dy, px, py, pz,
                                                        C.fl[t], L);
        br += ecl ? 0.0 : v;
    }
}

// Faces [t0, t1) of the block by groups: a run of 64, and its parts of 16 where
// the run is neither dark nor bright.
template <int LT, bool BEAM, bool GLENS, int STAR, bool ECL>
__device__ __forceinline__ void segment64(const Cols64 &C, const RunRec *sr, int t0, int t1,
                                          const Entry64 &E, const Arc64 &W, double zb,
                                          const Consts64 &L, double &br) {
    constexpr bool plain = !BEAM && !GLENS;
#pragma unroll 1
    for (int t = t0; t < t1;) {
        const int run = t / kRunFaces;
        const int re = (run + 1) * kRunFaces < t1 ? (run + 1) * kRunFaces : t1;
        int c = group64<ECL>(sr[kRunRecs * run], (float)zb, W);
        const bool whole = c == kGroupDark || (plain && c == kGroupBright);
#pragma unroll 1
        while (t < re) {
            int pe = re;
            if (!whole) {
                const int part = t / 16;
                pe = (part + 1) * 16 < re ? (part + 1) * 16 : re;
                c = group64<ECL>(sr[kRunRecs * run + 1 + (part & 3)], (float)zb, W);
            }
            if (c == kGroupDark) {
            } else if (plain && c == kGroupBright) {
                bright64<LT>(C, t, pe, E, L, br);
            } else if (ECL && c == kGroupRanges) {
                faces64<LT, BEAM, GLENS, STAR, ECL>(C, t, pe, E, zb, L, br);
            } else {
                faces64<LT, BEAM, GLENS, STAR, false>(C, t, pe, E, zb, L, br);
            }
            t = pe;
        }
    }
}

// Skipped or not, classified or not, every sum is bit-identical: what is left
// out are exact zeros and factors of one, and the faces keep their order. FP64
// issue bounds it (some 35 instructions for a visible element, 12 of them the
// square root). One entry a thread: the columns come from shared memory either
// way, a warp's arc is as narrow as it gets, and 32 warps an SM hide an element's
// chain; dark CTAs leave early, so smaller tiles also share the bright ones out.
// Curve of 100/200 strips and 15,000 entries, both stars at once, faces tested one
// by one at 4 entries and 128 threads 1.98 ms; by groups 1.75; 2 and 128 1.49,
// 1 and 128 1.51, 1 and 512 1.38, 1 and 256 1.34.
template <int LT, bool BEAM, bool GLENS, int STAR>
__global__ void __launch_bounds__(kThreads64, 4)
    k_flux64(FluxConsts k, FlatDev f, PhaseDev ph, double *part, int64_t ldp, DevStatus *st) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    constexpr bool need_pos = BEAM || GLENS;
    const int tid = threadIdx.x;
    const int64_t lo = (int64_t)blockIdx.y * kBlock;
    const int64_t n = f.n, n0 = *f.n0;
    const int64_t hi = (lo + kBlock < n) ? lo + kBlock : n;
    const bool need_ecl = hi > n0;
    constexpr uint32_t col = kBlock * 8, rec = kBlock / kRunFaces * kRunRecs * sizeof(RunRec);
    RunRec *sr = reinterpret_cast<RunRec *>(smem);
    double *s_dx = reinterpret_cast<double *>(smem + rec);
    double *s_dy = s_dx + kBlock, *s_dz = s_dy + kBlock, *s_fl = s_dz + kBlock;
    double *s_in = s_fl + kBlock, *s_out = s_in + kBlock;
    double *s_px = s_out + kBlock, *s_py = s_px + kBlock, *s_pz = s_py + kBlock;

    if (tid == 0) mbar_init(&bar, 1);
    __syncthreads();
    if (tid == 0) {
        uint32_t bytes = rec + 4 * col + (need_ecl ? 2 * col : 0u) + (need_pos ? 3 * col : 0u);
        mbar_arrive_expect_tx(&bar, bytes);
        bulk_g2s(sr, f.runs + kRunRecs * (lo / kRunFaces), rec, &bar);
        bulk_g2s(s_dx, f.dx + lo, col, &bar);
        bulk_g2s(s_dy, f.dy + lo, col, &bar);
        bulk_g2s(s_dz, f.dz + lo, col, &bar);
        bulk_g2s(s_fl, f.flux + lo, col, &bar);
        if (need_ecl) {
            bulk_g2s(s_in, f.in1 + lo, col, &bar);
            bulk_g2s(s_out, f.out1 + lo, col, &bar);
        }
        if (need_pos) {
            bulk_g2s(s_px, f.px + lo, col, &bar);
            bulk_g2s(s_py, f.py + lo, col, &bar);
            bulk_g2s(s_pz, f.pz + lo, col, &bar);
        }
    }
    const int64_t entry = (int64_t)blockIdx.x * kThreads64 + tid;
    // whole warps past the last entry leave (never the first, which waits for the
    // copies); threads past it in the last warp repeat it
    if ((entry & ~31ll) >= ph.nent) return;
    const int64_t e = entry < ph.nent ? entry : ph.nent - 1;
    const Entry64 E{ph.ex[e], ph.ey[e], ph.ez[e], ph.phin[e]};
    Arc64 W{(float)E.ex, (float)E.ey, (float)E.ez, 0.f, 0ull, 0ull};
    if (!(E.ex * E.ex + E.ey * E.ey + E.ez * E.ez < 1.000001)) W.ex = nanf("");
    W.exy = sqrtf(W.ex * W.ex + W.ey * W.ey);
    const unsigned long long pf = ph.pfx[e];
    warp_arc<1>(&pf, W.A, W.L);
    // the arc holds phases of one turn; with others among them ranges are tested singly
    if (!__all_sync(0xffffffffu, E.pn >= 0. && E.pn <= 1.)) {
        W.A = 0ull;
        W.L = ~0ull;
    }
    const Consts64 L{k.c[0], k.c[1], k.c[2], k.c[3], k.base, k.mucrit,
                     k.beam, k.spin, k.vfac, k.xcofm, k.rlens1};
    // a warp leaves together whether its copies arrived or the wait gave up,
    // so every lane reaches the votes below
    const bool staged = __all_sync(0xffffffffu, mbar_wait_bounded(&bar, 0));
    if (!staged) {
        if (tid == 0) {
            if (atomicCAS(&st->code, 0, 6) == 0) st->face = (int32_t)lo;
        }
        mbar_wait_bounded(&bar, 0);
        return;
    }
    const double zb = zero_below<BEAM>(L);
    const Cols64 C{s_dx, s_dy, s_dz, s_fl, s_in, s_out, s_px, s_py, s_pz};
    // plain segment, then one-range segment, counted from the block's first face
    const int64_t q0 = n0 - lo;
    const int end = (int)(hi - lo), q = q0 < 0 ? 0 : q0 < end ? (int)q0 : end;
    double br = 0.0;
    segment64<LT, BEAM, GLENS, STAR, false>(C, sr, 0, q, E, W, zb, L, br);
    segment64<LT, BEAM, GLENS, STAR, true>(C, sr, q, end, E, W, zb, L, br);
    if (entry < ph.nent) part[(int64_t)blockIdx.y * ldp + entry] = br;
}

// Several-range faces (the ragged segment of comp_light_flat.cpp:306-316):
// one thread per (face block, phase entry) continues the block's partial sum
// over the block's ragged faces in face order, each range tested in order.
// Element values come from the grid in Point order (the FlatGrid holds the
// same doubles): 64 faces at a time are gathered into shared memory, a thread
// each, so that the serial walk over them meets no chain of global loads (its
// index, then the face: 92 us for 10,000 faces and 2,000 entries, latency all
// of it; 31 staged). Then 32 faces at a time, a lane each, are held against all of
// the warp's entries; those left are summed two at a time without a
// vote: both stars of an opaque-disc model on 100/200 strips 96 -> 77 us.
constexpr int kRagTile = 64;
template <bool POS>
struct RagFace {
    double dx, dy, dz, flux;
    double2 r[kRagRanges];
    int32_t nr, pad_;
    double p[POS ? 3 : 1];
};

template <int LT, bool BEAM, bool GLENS, int STAR>
__global__ void __launch_bounds__(kThreadsRag)
    k_flux_ragged(FluxConsts k, FlatDev f, GridDev g, PhaseDev ph, int64_t blk, double *part,
                  int64_t ldp) {
    constexpr bool POS = BEAM || GLENS;
    __shared__ RagFace<POS> face[kRagTile];
    const int64_t b = blockIdx.y;
    const int64_t n = f.n, n1 = f.n1[0];
    const int64_t lo = b * blk, hi = (lo + blk < n) ? lo + blk : n;
    const int64_t c0 = lo > n1 ? lo : n1;
    if (c0 >= hi) return;
    // threads past the last entry repeat it without storing: warps stay whole
    // for the votes
    const int64_t e1 = blockIdx.x * (int64_t)kThreadsRag + threadIdx.x;
    const int64_t e = e1 < ph.nent ? e1 : ph.nent - 1;
    const Consts64 L{k.c[0], k.c[1], k.c[2], k.c[3], k.base, k.mucrit,
                     k.beam, k.spin, k.vfac, k.xcofm, k.rlens1};
    const double ex = ph.ex[e], ey = ph.ey[e], ez = ph.ez[e], pn = ph.phin[e];
    const unsigned long long pf = ph.pfx[e];
    unsigned long long A, La;
    warp_arc<1>(&pf, A, La);
    const int lane = threadIdx.x & 31;
    // every entry of the warp lies within wide of the middle lane's, or of the first one's
    // that is a number: a point whose time is not spoils no other
    const unsigned real = __ballot_sync(0xffffffffu, ex == ex && ey == ey && ez == ez);
    const int mid = ((real >> 16) & 1u) || !real ? 16 : __ffs(real) - 1;
    const double cx = __shfl_sync(0xffffffffu, ex, mid), cy = __shfl_sync(0xffffffffu, ey, mid),
                 cz = __shfl_sync(0xffffffffu, ez, mid);
    double wide = sqrt((ex - cx) * (ex - cx) + (ey - cy) * (ey - cy) + (ez - cz) * (ez - cz));
    for (int o = 16; o > 0; o >>= 1) wide = fmax(wide, __shfl_xor_sync(0xffffffffu, wide, o));
    wide = 1.0001 * wide + 1e-9;
    double acc = part[b * ldp + e];
    const double zb = zero_below<BEAM>(L);
    for (int64_t i0 = c0; i0 < hi; i0 += kRagTile) {
        const int m = (int)(hi - i0 < kRagTile ? hi - i0 : kRagTile);
        __syncthreads();
        if ((int)threadIdx.x < m) {
            const int64_t r = i0 + threadIdx.x - n1;
            const int32_t fi = f.ridx[r];
            RagFace<POS> &F = face[threadIdx.x];
            F.dx = g.nx[fi];
            F.dy = g.ny[fi];
            F.dz = g.nz[fi];
            F.flux = (double)g.flux[fi];
            F.nr = f.rn[r];
            for (int q = 0; q < kRagRanges; q++)  // past the last: hides nothing
                F.r[q] = q < F.nr ? f.rr[kRagRanges * r + q] : make_double2(10., -10.);
            if constexpr (POS) {
                F.p[0] = g.px[fi];
                F.p[1] = g.py[fi];
                F.p[2] = g.pz[fi];
            }
        }
        __syncthreads();
        for (int t0 = 0; t0 < m; t0 += 32) {
            // 32 faces, a lane each: turned away from, or hidden at, all of the warp's
            // entries; ranges that meet them
            int c = kGroupDark;
            if (t0 + lane < m) {
                const RagFace<POS> &F = face[t0 + lane];
                if (mu_of(cx, cy, cz, F.dx, F.dy, F.dz) + wide > zb)
                    c = ranges_class(F.r, F.nr, A, La);
            }
            unsigned todo = __ballot_sync(0xffffffffu, c != kGroupDark);
            const unsigned ranged = __ballot_sync(0xffffffffu, c == kGroupRanges);
            auto value = [&](int t) {
                const RagFace<POS> &F = face[t0 + t];
                const double mu = mu_of(ex, ey, ez, F.dx, F.dy, F.dz);
                bool ecl = false;
                if ((ranged >> t) & 1u) {
#pragma unroll
                    for (int q = 0; q < kRagRanges; q++) {
                        const double2 R = F.r[q];
                        ecl = ecl || (pn >= R.x && pn <= R.y) || pn <= R.y - 1.0;
                    }
                }
                double px = 0., py = 0., pz = 0.;
                if constexpr (POS) { px = F.p[0]; py = F.p[1]; pz = F.p[2]; }
                const double v = elem_mu<LT, BEAM, GLENS, STAR>(mu, ex, ey, ez, F.dx, F.dy, px, py,
                                                                pz, F.flux, L);
                return ecl ? 0.0 : v;
            };
            while (todo) {  // two at a time, added in order
                const int i = __ffs(todo) - 1;
                todo &= todo - 1u;
                const int j = todo ? __ffs(todo) - 1 : i;
                const double v = value(i), w = value(j);
                acc += v;
                if (todo) acc += w;
                todo &= todo - 1u;
            }
        }
    }
    if (e1 < ph.nent) part[b * ldp + e] = acc;
}

template <int LT, bool BEAM, bool GLENS, int STAR>
void launch_rag_t(const FluxConsts &k, const FlatDev &f, const GridDev &g, const PhaseDev &ph,
                  int64_t blk, int64_t nblk, double *part, int64_t ldp, cudaStream_t s) {
    dim3 grid((unsigned)((ph.nent + kThreadsRag - 1) / kThreadsRag), (unsigned)nblk);
    k_flux_ragged<LT, BEAM, GLENS, STAR><<<grid, kThreadsRag, 0, s>>>(k, f, g, ph, blk, part, ldp);
    count_launch();
}

template <int LT>
void launch_rag_lt(int star, const FluxConsts &k, const FlatDev &f, const GridDev &g,
                   const PhaseDev &ph, int64_t blk, int64_t nblk, double *part, int64_t ldp,
                   cudaStream_t s) {
    const bool beam = k.beam_on != 0, glens = (star == 1) && k.glens;
    if (star == 0) {
        if (beam) launch_rag_t<LT, true, false, 0>(k, f, g, ph, blk, nblk, part, ldp, s);
        else launch_rag_t<LT, false, false, 0>(k, f, g, ph, blk, nblk, part, ldp, s);
    } else if (glens) {
        if (beam) launch_rag_t<LT, true, true, 1>(k, f, g, ph, blk, nblk, part, ldp, s);
        else launch_rag_t<LT, false, true, 1>(k, f, g, ph, blk, nblk, part, ldp, s);
    } else {
        if (beam) launch_rag_t<LT, true, false, 1>(k, f, g, ph, blk, nblk, part, ldp, s);
        else launch_rag_t<LT, false, false, 1>(k, f, g, ph, blk, nblk, part, ldp, s);
    }
}

template <int LT, bool BEAM, bool GLENS, int STAR>
void launch_t(const FluxConsts &k, const FlatDev &f, const PhaseDev &ph, const FluxPlan &plan,
              double *part, int64_t ldp, DevStatus *st, cudaStream_t s) {
    constexpr bool need_pos = BEAM || GLENS;
    const size_t smem = (size_t)kBlock * 8 * (need_pos ? 9 : 6) +
                        kBlock / kRunFaces * kRunRecs * sizeof(RunRec);
    auto kern = k_flux64<LT, BEAM, GLENS, STAR>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dim3 grid((unsigned)plan.ntile, (unsigned)plan.nchunk);
    kern<<<grid, kThreads64, smem, s>>>(k, f, ph, part, ldp, st);
    count_launch();
}

template <int LT>
void launch_lt(int star, const FluxConsts &k, const FlatDev &f, const PhaseDev &ph,
               const FluxPlan &plan, double *part, int64_t ldp, DevStatus *st, cudaStream_t s) {
    const bool beam = k.beam_on != 0, glens = (star == 1) && k.glens;
    if (star == 0) {
        if (beam) launch_t<LT, true, false, 0>(k, f, ph, plan, part, ldp, st, s);
        else launch_t<LT, false, false, 0>(k, f, ph, plan, part, ldp, st, s);
    } else if (glens) {
        if (beam) launch_t<LT, true, true, 1>(k, f, ph, plan, part, ldp, st, s);
        else launch_t<LT, false, true, 1>(k, f, ph, plan, part, ldp, st, s);
    } else {
        if (beam) launch_t<LT, true, false, 1>(k, f, ph, plan, part, ldp, st, s);
        else launch_t<LT, false, false, 1>(k, f, ph, plan, part, ldp, st, s);
    }
}

// 8 independent DFMA chains per thread keep the FP64 pipe full.
__global__ void __launch_bounds__(256) k_dfma_probe(double *sink, int iters) {
    double a0 = threadIdx.x * 1e-3, a1 = a0 + 1., a2 = a0 + 2., a3 = a0 + 3.;
    double a4 = a0 + 4., a5 = a0 + 5., a6 = a0 + 6., a7 = a0 + 7.;
    const double m = 0.999999, c = 1e-6;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 16; u++) {
            a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
            a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
        }
    }
    const double r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (r == 12345.) sink[0] = r;  // keeps the chains live
}

}  // namespace

void launch_dfma_probe(double *sink, int blocks, int iters, double *gflop, cudaStream_t s) {
    k_dfma_probe<<<blocks, 256, 0, s>>>(sink, iters);
    *gflop = 2.0 * 8 * 16 * (double)iters * 256.0 * blocks * 1e-9;
}

void launch_flux_ragged(int star, const FluxConsts &k, const FlatDev &f, const GridDev &g,
                        const PhaseDev &ph, int64_t blk, int64_t nblk, double *part,
                        int64_t ldp, cudaStream_t s) {
    if (ph.nent <= 0 || nblk <= 0 || !f.n1) return;
    if (k.ltype == 1) launch_rag_lt<1>(star, k, f, g, ph, blk, nblk, part, ldp, s);
    else launch_rag_lt<0>(star, k, f, g, ph, blk, nblk, part, ldp, s);
}

void launch_flux64(int star, const FluxConsts &k, const FlatDev &f, const PhaseDev &ph,
                   const FluxPlan &plan, double *part, int64_t ldp, DevStatus *st,
                   cudaStream_t s) {
    if (k.ltype == 1) launch_lt<1>(star, k, f, ph, plan, part, ldp, st, s);
    else launch_lt<0>(star, k, f, ph, plan, part, ldp, st, s);
}

}  // namespace lcg
