// The engine's host side (engine.cu, batch_host.cu) on the CPU, with allocations that fail.
//
// Neither holds device code: they are compiled here with the host compiler against a
// runtime in which device memory is host memory and the n-th allocation of a call returns
// cudaErrorMemoryAllocation. The kernels' launchers are replaced by checks of what they are
// given: that every array lives and is large enough, that the ring table belongs to
// the grid, and that a sweep reads the fluxes of the model it is launched for.
//
//   host_check rings|cache|data|pin|first|batch|moved   (stdin: lcg_model A, lcg_model B)
//
// pin: many contexts and calls with A, counting pinned blocks. first: prints the device allocations of 2 MB
// or more of a context's first call, with A. batch: batched calls in place of single ones.
// moved: a batch's captured graph after its points moved. The others:
// A call with A, one with B whose k-th allocation fails, then A again (mode data: points for
// the first call, more of them for the second), in a new context for every k until the second
// call has none left to fail. Prints the number of failures tried and of what was wrong;
// exits 1 if anything was.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>

#include "../../lcurve_re_b200/csrc/engine.cu"
#include "../../lcurve_re_b200/csrc/batch_host.cu"

static std::map<char *, size_t> g_mem;
static long g_countdown = -1;  // allocations until one fails
static int g_wrong = 0, g_pinned = 0, g_pins = 0, g_large = 0;
static const lcg_model *g_model = nullptr;
static std::map<const void *, double> g_flux_t, g_flat_t;  // by array: the model's temperature

static void wrong(const char *what) {
    g_wrong++;
    fprintf(stderr, "wrong: %s\n", what);
}
static size_t room(const void *p) {  // bytes left in the allocation that p points into
    auto it = g_mem.upper_bound((char *)p);
    if (!p || it == g_mem.begin()) return 0;
    --it;
    const size_t at = (size_t)((char *)p - it->first);
    return at < it->second ? it->second - at : 0;
}
template <class T>
static void need(const T *p, int64_t n, const char *what) {
    if (room(p) < (size_t)n * sizeof(T)) wrong(what);
}
// what a captured stream would run when its graph is launched
static std::vector<std::function<void()>> g_graph;
static bool g_capturing = false;
template <class F>
static void stream(F f) {
    if (g_capturing) g_graph.push_back(f);
    else f();
}
static const size_t kKeep = 1 << 20;
static char *g_arena = nullptr;      // blocks of kKeep bytes, given out lowest address first
static std::set<char *> g_free;
static cudaError_t get(void **p, size_t n) {
    if (g_countdown > 0 && --g_countdown == 0) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    if (g_arena && n <= kKeep && !g_free.empty()) {
        *p = *g_free.begin();
        g_free.erase(g_free.begin());
    } else {
        *p = calloc(1, n);
    }
    g_mem[(char *)*p] = n;
    return cudaSuccess;
}
static cudaError_t drop(void *v) {
    char *p = (char *)v;
    g_mem.erase(p);
    if (g_arena && p >= g_arena && p < g_arena + 64 * kKeep) g_free.insert(p);
    else free(p);
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    g_large += n >= (size_t)2 << 20;
    return get(p, n);
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    g_pinned++;
    g_pins++;
    return get(p, n);
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) {
    g_pinned++;
    g_pins++;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void *) {
    g_pinned--;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { return drop(p); }
cudaError_t cudaFreeHost(void *p) {
    g_pinned--;
    return drop(p);
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    stream([=] {
        if (room(k == cudaMemcpyHostToDevice ? d : s) < n) wrong("a copy past its array");
        else memcpy(d, s, n);
    });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind,
                              cudaStream_t) {
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    stream([=] {
        if (room(p) < n) wrong("a clear past its array");
        else memset(p, v, n);
    });
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    g_capturing = true;
    g_graph.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    g_capturing = false;
    *g = (cudaGraph_t)&g_graph;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) {
    *e = (cudaGraphExec_t)g;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    for (auto &f : g_graph) f();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0.f; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "allocation failed by the test"; }
}

namespace lcg {

static void need_grid(const GridDev &g) {
    for (const double *p : {g.px, g.py, g.pz, g.nx, g.ny, g.nz, g.ein, g.eout}) need(p, g.n, "grid");
    for (const float *p : {g.area, g.grav}) need(p, g.n, "grid");
    if (g.flux) need(g.flux, g.n, "grid");  // batches keep none
    need(g.necl, g.n, "grid");
}
void launch_grid(const GridParams &p, const RingRec *r, GridDev g, int32_t *cnt, DevStatus *,
                 cudaStream_t) {
    need_grid(g);
    need(cnt, 8, "counters");
    if (room(r) < (size_t)p.nrings * sizeof(RingRec) || p.nrings < 1) {
        wrong("a ring table shorter than its grid's rings");
        return;
    }
    const RingRec &last = r[p.nrings - 1];
    if (last.off + last.nphi != g.ntiled || last.hoff + (last.nphi + 1) / 2 != p.nhalf)
        wrong("a ring table of another grid");
    if (llabs(g.n - g.ntiled) > 4) wrong("a face count of another grid");
}
void launch_eclipse(const EclParams &, int32_t, GridDev g, int32_t *q, int32_t *c, double4 *es,
                    int32_t *h, DevStatus *, int, int32_t, cudaStream_t) {
    need_grid(g);
    need(q, g.n, "queue"); need(c, 8, "counters"); need(es, g.n, "states"); need(h, g.n, "hits");
}
int64_t cont_blocks(int64_t n) { return (n + 255) / 256; }
void launch_continuum(const ContParams &p, GridDev g, int32_t *cnt, double *dsum, cudaStream_t) {
    need_grid(g);
    if (cnt) need(cnt, 2 * cont_blocks(g.n), "counts");
    if (dsum) need(dsum, 4 * cont_blocks(g.n), "sums");
    g_flux_t[g.flux] = p.t_own;
}
void launch_flatten(GridDev g, FlatDev f, const int32_t *cnt, int mixed, int need_pos,
                    const FastCoef &fc, cudaStream_t) {
    need_grid(g);
    need(cnt, 2 * cont_blocks(g.n), "counts");
    if (need_pos && mixed) need(f.pos, f.npad, "positions");
    if (mixed && fc.on) need(f.fp, 8 * f.npad, "records");
    g_flat_t[f.n0] = g_flux_t[g.flux];
}
void launch_phases(const PhaseParams &, const DatumRec *d, const int64_t *off, int32_t n, PhaseDev ph,
                   bool, V3, double, cudaStream_t) {
    need(d, n, "points");
    need(off, n + 1, "offsets");
    if (room(off) >= (size_t)(n + 1) * 8 && off[n] > ph.nent) wrong("entries of other points");
    for (const double *p : {ph.ex, ph.ey, ph.ez, ph.phin, ph.w1, ph.w2}) need(p, ph.nent, "entries");
}
void launch_scatter(const ScatterParams &, const ReduceParams &, const PhaseDev &, const DatumRec *d,
                    const int64_t *, int32_t n, double *calc, cudaStream_t) {
    need(d, n, "points");
    need(calc, n, "curve");
}
void launch_finalize(int32_t, const DatumRec *, int32_t, double *, double, const TailIn &, TailOut *,
                     cudaStream_t) {}
void launch_tail(const TailIn &, TailOut *, cudaStream_t) {}
void launch_interp(const DatumRec *, int32_t, const int64_t *, int32_t, const double *, double *,
                   int32_t, double *, cudaStream_t) {}
void launch_iscale(int32_t, int32_t, const DatumRec *, int32_t, const double *, double *, double *,
                   double *, double *, cudaStream_t) {}
void launch_pack_flat(FlatDev, int64_t, int, cudaStream_t) {}
void launch_pack_phases(PhaseDev, cudaStream_t) {}
void launch_run_bounds64(const FlatDev &, cudaStream_t) {}
void launch_run_bounds_geo(const FlatDev &, cudaStream_t) {}
FluxPlan plan_flux(int mixed, int fast, int64_t nface, int64_t nent, int) {
    FluxPlan p{};
    p.fast = mixed && fast;
    p.ppt = 1;
    p.threads = 256;
    p.chunk = p.group = 1024;
    p.nchunk = (nface + 1023) / 1024;
    p.ntile = (nent + 255) / 256;
    return p;
}
void launch_flux(int mixed, int star, const FluxConsts &, const FlatDev &f, const PhaseDev &,
                 const FluxPlan &, double *part, int64_t ldp, DevStatus *, cudaStream_t) {
    if (mixed) need(f.ecl, f.npad, "ranges");
    need(part, ldp, "partial sums");
    if (g_flat_t[f.n0] != (star == 0 ? g_model->t1 : g_model->t2))
        wrong("a sweep over another model's fluxes");
}
void launch_flux_ragged(int, const FluxConsts &, const FlatDev &, const GridDev &, const PhaseDev &,
                        int64_t, int64_t, double *, int64_t, cudaStream_t) {}
void launch_components(const CompParams &, ElemRec *, double4 *, DevStatus *, cudaStream_t) {}
void launch_disc_faces(const DiscGeom &, const GridDev &, uint8_t *, double2 *, int32_t *, DevStatus *,
                       cudaStream_t) {}
void launch_comp_sums(const ElemRec *, int32_t, int32_t, int32_t, double, double, PhaseDev const &,
                      double *, double *, int64_t, cudaStream_t) {}
int64_t comp_sums_scratch(int32_t, int64_t) { return 1; }
void launch_fma_probe(float *, int, int, double *, cudaStream_t) {}
void launch_dfma_probe(double *, int, int, double *, cudaStream_t) {}
void launch_batch_grid(const BatchDev &b, int, cudaStream_t) {
    stream([=] {
        for (int k = 0; k < b.counts[0]; k++) {
            const SlotDev &S = b.slots[b.geo_slot[k]];
            const RingRec *r = b.rings + S.ring0;
            if (room(r) < (size_t)S.gp.nrings * sizeof(RingRec)) {
                wrong("a ring pool shorter than a slot's rings");
                continue;
            }
            const RingRec &last = r[S.gp.nrings - 1];
            if (last.off + last.nphi != S.ntiled) wrong("a ring table of another slot");
        }
    });
}
void launch_batch_eclipse(const BatchDev &b, int, int32_t, cudaStream_t) {
    stream([=] {
        need_grid(b.g);
        need(b.queue, b.qcap, "queue");
        need(b.es, b.qcap, "states");
    });
}
void launch_batch_partition(const BatchDev &, int, cudaStream_t) {}
void launch_batch_continuum(const BatchDev &b, int, cudaStream_t) {
    stream([=] { need(b.fp, 8 * b.g.n, "records"); });
}
void launch_batch_phases(const BatchDev &, const DatumRec *d, const int64_t *off, int32_t n,
                         const BatchPhases &, cudaStream_t) {
    stream([=] {
        need(d, n, "points");
        need(off, n + 1, "offsets");
        if (room(off) >= (size_t)(n + 1) * 8 && (off[0] != 0 || off[n] != n)) wrong("other offsets");
    });
}
void launch_batch_flux(const BatchDev &, const BatchPhases &, const FluxPlan &, double *, int64_t,
                       cudaStream_t) {}
void launch_batch_reduce(const BatchDev &, const BatchPhases &, const double *, int64_t, double *,
                         const DatumRec *d, const int64_t *off, int32_t n, int32_t, double *, double *,
                         double *, cudaStream_t) {
    stream([=] {
        need(d, n, "points");
        need(off, n + 1, "offsets");
    });
}
void launch_gather_rows(const double *, int32_t, const int32_t *, int32_t, double *, cudaStream_t) {}
namespace eng {
bool comp_setup(const lcg_model &, CompParams &, std::vector<DiscRing> &, Fail &) { return false; }
}  // namespace eng
}  // namespace lcg

static lcg_status points(lcg_ctx *c, int n) {
    std::vector<lcg_datum> d((size_t)n);
    memset(d.data(), 0, d.size() * sizeof(lcg_datum));
    for (int i = 0; i < n; i++) {
        d[i].time = 1e-3 * i;
        d[i].ferr = d[i].weight = 1.;
        d[i].ndiv = 1;
    }
    return lcg_set_data(c, d.data(), n);
}
static lcg_status curve(lcg_ctx *c, const lcg_model &m, int n) {
    std::vector<double> calc((size_t)n);
    double sfac[5] = {1., 1., 1., 1., 1.}, out[LCG_NOUT];
    g_model = &m;
    return lcg_light_curve_resident(c, &m, 0, sfac, calc.data(), out);
}

static lcg_status batch(lcg_ctx *c, const lcg_model &a, const lcg_model &b, int n) {
    lcg_model m[2] = {a, b};
    std::vector<double> calc(2 * (size_t)n);
    double sfac[10], chisq[2], wnok[2];
    int32_t st[2];
    for (double &s : sfac) s = 1.;
    // new temperatures: nothing is reused
    static double step = 0.;
    m[0].t1 += (step += 1.);
    m[1].t1 += step;
    return lcg_light_curve_batch_resident(c, m, 2, 0, sfac, calc.data(), chisq, wnok, st);
}

int main(int argc, char **argv) {
    lcg_model a, b;
    if (argc < 2 || fread(&a, sizeof a, 1, stdin) != 1 || fread(&b, sizeof b, 1, stdin) != 1) return 2;
    if (!strcmp(argv[1], "first")) {
        lcg_ctx *c = nullptr;
        if (lcg_create(&c, nullptr) || points(c, 100) || curve(c, a, 100)) return 3;
        printf("%d %d\n", g_large, g_wrong);
        lcg_destroy(c);
        return g_wrong ? 1 : 0;
    }
    if (!strcmp(argv[1], "pin")) {
        // contexts one after another and side by side share one block
        lcg_ctx *c[20];
        for (int i = 0; i < 50; i++) {
            if (lcg_create(&c[0], nullptr) || points(c[0], 5000) || curve(c[0], a, 5000)) return 3;
            lcg_destroy(c[0]);
        }
        if (g_pins != 1) wrong("more than one block pinned, or none");
        // 15 pages each of 256: the block is full with the 17th
        for (lcg_ctx *&x : c)
            if (lcg_create(&x, nullptr) || points(x, 5000) || curve(x, a, 5000)) return 3;
        std::set<const void *> at;
        for (lcg_ctx *x : c) at.insert(x->h_in.p), at.insert(x->h_res.p);
        if (at.size() != 40) wrong("two contexts in the same pages");
        if (!c[0]->h_in.pooled || c[19]->h_in.pooled) wrong("the block's size");
        if (g_pins != 1) wrong("pinned memory before it can pay");
        for (int i = 0; i < 400; i++)
            if (points(c[19], 5000) || curve(c[19], a, 5000)) return 3;
        if (!c[19]->h_in.pinned) wrong("a block that has paid for it, not pinned");
        for (lcg_ctx *x : c) lcg_destroy(x);
        if (g_pinned != 1) wrong("pinned memory left behind");
        if (lcg_create(&c[0], nullptr) || points(c[0], 80000) || !c[0]->h_in.pooled)
            wrong("pages not given back");
        if (points(c[0], 200000) || c[0]->h_in.pooled) wrong("more than the block holds");
        lcg_destroy(c[0]);
        printf("%d %d\n", g_pins, g_wrong);
        return g_wrong ? 1 : 0;
    }
    if (!strcmp(argv[1], "moved")) {
        // three blocks in a row, the points in the first and the offsets in the third; then the
        // second becomes free, and larger points get the first and the second
        lcg_ctx *c = nullptr;
        if (lcg_create(&c, nullptr)) return 3;
        g_arena = (char *)calloc(64, kKeep);
        for (int i = 0; i < 64; i++) g_free.insert(g_arena + i * kKeep);
        void *blk[3];
        for (void *&p : blk) cudaMalloc(&p, 64);
        cudaFree(blk[0]);
        cudaFree(blk[2]);
        if (points(c, 100) || c->data.p != blk[0] || (void *)c->off.p != blk[2]) return 4;
        for (int i = 0; i < 3; i++)
            if (batch(c, a, a, 100)) return 3;
        cudaFree(blk[1]);
        if (points(c, 5000) || c->data.p != blk[0] || (void *)c->off.p != blk[1]) return 4;
        if (points(c, 100) || batch(c, a, a, 100)) return 3;
        lcg_destroy(c);
        printf("1 %d\n", g_wrong);
        return g_wrong ? 1 : 0;
    }
    const bool data = !strcmp(argv[1], "data"), many = !strcmp(argv[1], "batch");
    int k = 1;
    for (;; k++) {
        lcg_ctx *c = nullptr;
        if (lcg_create(&c, nullptr) || points(c, 100)) return 3;
        for (int i = 0; i < (many ? 3 : 1); i++)
            if (many ? batch(c, a, a, 100) : curve(c, a, 100)) return 3;
        g_countdown = k;
        const lcg_status st = data ? points(c, 5000) : many ? batch(c, a, b, 100) : curve(c, b, 100);
        const bool failed = g_countdown == 0;
        g_countdown = -1;
        if (failed != (st != LCG_OK)) wrong("a failed allocation without a status");
        lcg_status again = many ? batch(c, a, b, 100) : curve(c, a, 5000);
        for (int i = 0; i < 3 && many && !again; i++) again = batch(c, i ? b : a, a, 100);
        // after points that were not taken there are none
        if (data ? (again == LCG_OK) == failed : again != LCG_OK) {
            wrong("the call after it");
            fprintf(stderr, "  %s\n", lcg_last_error(c));
        }
        lcg_destroy(c);
        if (!failed) break;
    }
    printf("%d %d\n", k - 1, g_wrong);
    return g_wrong ? 1 : 0;
}
