// extern "C" entry points of libwadi_b200 (declared in include/wadi_b200.h) and the host side of the handle.
//
// The handle binds caller-owned device buffers; the only memory it allocates is its own host record (with a pinned copy
// of the run table for the loop's read-back) and the CUDA graphs of the device loop. Ping-pong pairs (h, u, v, mx, my) are
// resolved through the handle's parity, which flips after every step: the reference swaps its arrays the same way (wadi2d/solver/gpu/backend.py:185-188).
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>

#include <cuda.h>

#include "w2b_common.cuh"
#include "w2b_tma.cuh"

namespace w2b {
// The face and update passes of w2b_step.cu, built twice: exact (the reference's float32 bits) and fast.
#define W2B_PASSES_DECL                                                             \
    cudaError_t faces_setup();                                                      \
    void launch_probe(const StepArgs& A, int t, float dt, float* out, cudaStream_t s); \
    int faces_occupancy();                                                          \
    void launch_faces(const TMaps& M, const StepArgs& A, int grid, cudaStream_t s); \
    cudaError_t update_setup();                                                     \
    int update_occupancy();                                                         \
    void launch_update(const TMaps& M, const StepArgs& A, int grid, int control, cudaStream_t s); \
    int strips_occupancy(int rows);                                                 \
    void launch_strips(int rows, const TMaps& M, const StepArgs& A, int grid, cudaStream_t s); \
    cudaError_t resident_setup();                                                   \
    int resident_occupancy(int rows);                                               \
    cudaError_t launch_resident(int rows, const ResidentMaps& M, const StepArgs& A, int grid, int occupancy, \
                                int max_steps, const HostStep& host, cudaStream_t s);
namespace exact {
W2B_PASSES_DECL
}
namespace fast {
W2B_PASSES_DECL
}
#undef W2B_PASSES_DECL

struct Passes {
    cudaError_t (*faces_setup)();
    void (*launch_probe)(const StepArgs&, int, float, float*, cudaStream_t);
    int (*faces_occupancy)();
    void (*launch_faces)(const TMaps&, const StepArgs&, int, cudaStream_t);
    cudaError_t (*update_setup)();
    int (*update_occupancy)();
    void (*launch_update)(const TMaps&, const StepArgs&, int, int, cudaStream_t);
    int (*strips_occupancy)(int);
    void (*launch_strips)(int, const TMaps&, const StepArgs&, int, cudaStream_t);
    cudaError_t (*resident_setup)();
    int (*resident_occupancy)(int);
    cudaError_t (*launch_resident)(int, const ResidentMaps&, const StepArgs&, int, int, int, const HostStep&,
                                   cudaStream_t);
};
static const Passes EXACT_PASSES = {exact::faces_setup,  exact::launch_probe,     exact::faces_occupancy,
                                    exact::launch_faces, exact::update_setup,     exact::update_occupancy,
                                    exact::launch_update, exact::strips_occupancy, exact::launch_strips,
                                    exact::resident_setup, exact::resident_occupancy, exact::launch_resident};
static const Passes FAST_PASSES = {fast::faces_setup,  fast::launch_probe,     fast::faces_occupancy,
                                   fast::launch_faces, fast::update_setup,     fast::update_occupancy,
                                   fast::launch_update,  fast::strips_occupancy,  fast::launch_strips,
                                   fast::resident_setup, fast::resident_occupancy, fast::launch_resident};
static const Passes& passes(const W2BParams& P) { return P.arith == W2B_ARITH_FAST ? FAST_PASSES : EXACT_PASSES; }

void launch_cbrt_check(uint32_t first, uint32_t count, unsigned long long* out, cudaStream_t s);
void launch_wait_check(uint32_t polls, long long* out, cudaStream_t s);
void launch_momentum(const StepArgs& A, int sms, cudaStream_t s);
void launch_asleep(const StepArgs& A, int sms, cudaStream_t s);
__global__ void boundary_kernel(StepArgs A);
__global__ void step_end_kernel(StepArgs A);
__global__ void rebuild_kernel(const __grid_constant__ StepArgs A, int adopt);
__global__ void begin_kernel(const __grid_constant__ StepArgs A, Ctl c, W2BClock one, double t_end, long long max_steps,
                             const W2BClock* clocks, const double* t_ends);
__global__ void setstep_kernel(StepArgs A, float dtf, int want_wave, int want_wet, int nact);
__global__ void plan_kernel(StepArgs A, const int32_t* list, int count);
__global__ void maxima_kernel(StepArgs A, float time, float arrive, float deep, int nact);
__global__ void tally_kernel(StepArgs A, double dt);
__global__ void ref_to_native_kernel(const float* ref, float* nat, const int32_t* tiles, int ntiles, int px);
__global__ void native_to_ref_kernel(const float* nat, float* ref, const int32_t* tiles, const int32_t* tile_of,
                                     int ntiles, int ny, int nx, int px);
__global__ void pack_tables_kernel(const float* dtab, const float* ftabx, const float* ftaby, float2* dtab2,
                                   float4* fx, float4* fy, int ntiles, int rows);
__global__ void bmark_kernel(StepArgs A, int clear_words);
__global__ void active_flags_kernel(StepArgs A, int n);

// A launch configuration of the device loop: the face pass's form (whole tiles, or the strip form: half tiles in
// smaller CTAs), its CTAs a SM, the update pass's CTAs a SM, and loop steps a launch: a captured graph of the passes'
// kernels, or (resident) one cooperative launch that takes the steps itself, with the strip form's units. Every
// configuration computes the same bits (a face's arithmetic does not depend on the form or the grid, and the wave
// maximum is an order-free integer max); they differ only in time.
struct LoopConfig {
    int faces_per_sm, update_per_sm, steps;
    int strips;  // the face pass's form: 0 whole tiles, else strips of this many rows (16 or 8)
    int resident;
};
constexpr int TUNE_CANDIDATES = 7;  // the default, it with more steps a graph, two strip forms, three resident ones
constexpr int FORCED = TUNE_CANDIDATES;          // the slot of a configuration the caller fixes
constexpr int TAILS = 2, TAIL_STEPS[TAILS] = {4, 1};  // graphs of fewer steps, for the end of a call
constexpr int TUNE_SAMPLES = 3;                  // timed launches a candidate before the tuner settles
constexpr int MAX_GRAPH_STEPS = 64;
constexpr double TUNE_MARGIN = 0.02;

// The device loop's captured graphs, one a configuration, and the online tuner that picks among them: while tuning,
// successive graph launches rotate through the candidates, each timed with CUDA events on the launching stream from
// the end of the graph before it (so the host's read of the clocks between graphs counts against the configuration
// whose graph follows it) and divided by the loop steps that ran (the empty steps of a graph that outlasts its runs
// count against the configuration that spent them). Once every candidate has TUNE_SAMPLES launches, the fastest per
// loop step is kept, the default unless another beats it by more than TUNE_MARGIN.
struct Loop {
    LoopConfig cand[TUNE_CANDIDATES + 1];
    int ncand = 0;
    cudaGraphExec_t exec[TUNE_CANDIDATES + 1][TAILS + 1] = {};  // of the configuration's steps, and of TAIL_STEPS'
    unsigned version[TUNE_CANDIDATES + 1][TAILS + 1];
    double sec[TUNE_CANDIDATES] = {};
    long long steps[TUNE_CANDIDATES] = {};
    int samples[TUNE_CANDIDATES] = {};
    int next = 0, chosen = 0;
    int tuning = 1;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};  // a launch's start; the ends of two successive launches
    Loop() {
        for (auto& v : version)
            for (auto& w : v) w = ~0u;
    }
};

constexpr int RESIDENT_ROWS[3] = {16, 8, 4};  // the resident loop's strip heights
static int resident_index(int rows) { return rows == 16 ? 0 : (rows == 8 ? 1 : 2); }

struct Handle {
    W2BGridDesc g{};
    W2BLayout L{};
    W2BParams P{};
    W2BBuffers B{};
    int cur = 0;  // run 0's current half (the device keeps it in R.parity[0])
    int nact = 0;
    bool touched = false;  // a state array has been in a caller's hands since the last step (asleep_kernel)
    int nruns = 1;
    RunTab R;
    int nb = 0;
    const int32_t *bcell = nullptr, *bref = nullptr, *bkind = nullptr;
    const float *bd0 = nullptr, *bh0 = nullptr;
    int ntally = 0;
    const int32_t *tface = nullptr, *taxis = nullptr;
    const float* tsign = nullptr;
    double* ttotal = nullptr;
    int nlines = 0;
    const int32_t *lstart = nullptr, *lface = nullptr, *laxis = nullptr;
    const float* lsign = nullptr;
    double *lq = nullptr, *lpeak = nullptr, *ltime = nullptr;
    int sms = 148;
    int step_blocks = 148;   // resident CTAs of the update pass
    int faces_blocks = 296;  // resident CTAs of the face pass
    int faces_occ = 2, update_occ = 1;  // resident CTAs a SM of the two passes
    int strips16_occ = 4, strips8_occ = 8;  // resident CTAs a SM of the face pass's strip forms
    int resident_occ[3] = {1, 1, 1};  // and of the resident loop's, in the order of RESIDENT_ROWS
    char* host = nullptr;  // pinned: the run table and the control block as read back, and a batch's clocks and ends
    TMaps tmaps;
    ResidentMaps rmaps[3];
    unsigned version = 0;   // bumped whenever a graph would capture stale arguments
    Loop loop;
    cudaStream_t cap = nullptr;  // private stream the loop graphs are captured on (a legacy stream cannot be)
    Ctl* ctl() const { return reinterpret_cast<Ctl*>(B.ctl); }
};

static StepArgs make_args(const Handle& H) {
    StepArgs A;
    memset(&A, 0, sizeof(A));
    A.P = H.P;
    A.rows = H.g.rows;
    A.px = H.L.px;
    A.ntiles = H.g.ntiles;
    A.nty = H.g.ny / TILE;
    A.ntx = H.g.nx / TILE;
    for (int q = 0; q < 2; ++q) {
        A.hh[q] = H.B.h[q];
        A.uu[0][q] = H.B.u[q];
        A.uu[1][q] = H.B.v[q];
        A.mm[0][q] = H.B.mx[q];
        A.mm[1][q] = H.B.my[q];
    }
    A.d = H.B.d;
    A.q[0] = H.B.qx;
    A.q[1] = H.B.qy;
    A.q1[0] = H.B.qx1;
    A.q1[1] = H.B.qy1;
    A.res = H.B.res;
    A.src = H.B.src;
    A.om = H.B.om;
    A.zc[0] = H.B.zcx;
    A.zc[1] = H.B.zcy;
    A.hc = H.B.hc;
    for (int a = 0; a < 2; ++a) {
        A.fl[a] = H.B.fl[a];
        A.fr[a] = H.B.fr[a];
        A.gl[a] = H.B.gl[a];
        A.gr[a] = H.B.gr[a];
        A.ef[a] = H.B.ef[a];
        A.cw[a] = H.B.cw[a];
        A.ftab4[a] = reinterpret_cast<const float4*>(H.B.ftab4[a]);
    }
    A.dtab2 = reinterpret_cast<const float2*>(H.B.dtab2);
    A.table_tile = H.B.table_tile;
    A.tiles = H.B.tiles;
    A.tile_of = H.B.tile_of;
    A.nbr = H.B.nbr;
    A.active = H.B.active;
    A.wave = H.B.wave;
    A.wet = H.B.wet;
    A.keep = H.B.keep;
    A.idle = H.B.idle;
    A.is_act = H.B.is_act;
    A.woken = H.B.woken;
    A.work = H.B.work;
    A.list = H.B.active;  // the host-driven step takes the active list; the device loop its work list
    A.scratch = H.B.scratch;
    for (int e = 0; e < 5; ++e) A.env[e] = H.B.env[e];
    A.bmark = H.B.bmark;
    A.nb = H.nb;
    A.bcell = H.bcell;
    A.bref = H.bref;
    A.bkind = H.bkind;
    A.bd0 = H.bd0;
    A.bh0 = H.bh0;
    A.ntally = H.ntally;
    A.tface = H.tface;
    A.taxis = H.taxis;
    A.tsign = H.tsign;
    A.ttotal = H.ttotal;
    A.nlines = H.nlines;
    A.lstart = H.lstart;
    A.lface = H.lface;
    A.laxis = H.laxis;
    A.lsign = H.lsign;
    A.lq = H.lq;
    A.lpeak = H.lpeak;
    A.ltime = H.ltime;
    A.ctl = H.ctl();
    A.any = &A.ctl->any;
    A.any_next = &A.ctl->any2;
    A.tile_run = H.B.tile_run;
    A.lpair = reinterpret_cast<float2*>(H.B.lpair);
    A.lrow = H.B.lrow;
    A.R = H.R;
    A.nruns = H.nruns;
    return A;
}

bool handle_args(void* handle, StepArgs* out) {
    if (!handle || !out) return false;
    *out = make_args(*static_cast<Handle*>(handle));
    return true;
}

static int cuda_status(cudaError_t e, const char* where) {
    if (e == cudaSuccess) return W2B_OK;
    fprintf(stderr, "libwadi_b200: %s: %s\n", where, cudaGetErrorString(e));
    return W2B_ECUDA;
}

#define CK(call)                                              \
    do {                                                      \
        int s_ = cuda_status((call), #call);                  \
        if (s_ != W2B_OK) return s_;                          \
    } while (0)
#define CKL(where) CK(cudaGetLastError())

static int blocks_for(const Handle& H, int n) { return n < H.step_blocks ? (n > 0 ? n : 1) : H.step_blocks; }
static int faces_grid(const Handle& H, int n) { return n < H.faces_blocks ? (n > 0 ? n : 1) : H.faces_blocks; }

// cuTensorMapEncodeTiled, fetched from the driver at run time (so the library does not link libcuda).
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int encode_2d(EncodeTiled enc, CUtensorMap* map, const float* base, const W2BGridDesc& g, const W2BLayout& L,
                     uint32_t bw, uint32_t bh) {
    if (!base || ((uintptr_t)base & 15)) return W2B_EINVAL;
    const cuuint64_t dims[2] = {(cuuint64_t)L.px, (cuuint64_t)(g.ny + 2 * L.gy)};
    const cuuint64_t strides[1] = {(cuuint64_t)L.px * 4};
    const cuuint32_t box[2] = {bw, bh};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fprintf(stderr, "libwadi_b200: cuTensorMapEncodeTiled failed (%d)\n", (int)r);
        return W2B_ECUDA;
    }
    return W2B_OK;
}

static int build_tmaps(Handle& H) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
        q != cudaDriverEntryPointSuccess)
        return W2B_ECUDA;
    EncodeTiled enc = reinterpret_cast<EncodeTiled>(fn);
    const W2BBuffers& B = H.B;
    int st = W2B_OK;
    auto box = [&](CUtensorMap* m, const float* p) {
        if (st == W2B_OK) st = encode_2d(enc, m, p, H.g, H.L, 40, 36);
    };
    auto own = [&](CUtensorMap* m, const float* p) {
        if (st == W2B_OK) st = encode_2d(enc, m, p, H.g, H.L, 32, 32);
    };
    box(&H.tmaps.tile.d, B.d);
    box(&H.tmaps.tile.qx, B.qx);
    box(&H.tmaps.tile.qy, B.qy);
    box(&H.tmaps.tile.om, B.om);
    box(&H.tmaps.tile.zcx, B.zcx);
    box(&H.tmaps.tile.zcy, B.zcy);
    box(&H.tmaps.update.qx1, B.qx1);
    box(&H.tmaps.update.qy1, B.qy1);
    own(&H.tmaps.update.res, B.res);
    own(&H.tmaps.update.src, B.src);
    for (int p = 0; p < 2; ++p) {
        box(&H.tmaps.tile.h[p], B.h[p]);
        box(&H.tmaps.update.h[p], B.h[p]);
        box(&H.tmaps.tile.u[p], B.u[p]);
        box(&H.tmaps.tile.v[p], B.v[p]);
        own(&H.tmaps.tile.mx[p], B.mx[p]);
        own(&H.tmaps.tile.my[p], B.my[p]);
    }
    // the strip forms' boxes, 40 columns of the rows the face arithmetic reads around a strip of `rows` rows: the
    // velocities rows + 4 (two above, two below), the y discharge rows + 2, the x lip rows, depth, mean depth, x
    // discharge and y lip rows + 1 (one above); 32 x rows for the momenta
    for (const int rows : RESIDENT_ROWS) {
        StripMaps& S = H.rmaps[resident_index(rows)].s;
        auto strip = [&](CUtensorMap* m, const float* q, int extra) {
            if (st == W2B_OK) st = encode_2d(enc, m, q, H.g, H.L, 40, (uint32_t)(rows + extra));
        };
        auto strip_own = [&](CUtensorMap* m, const float* q) {
            if (st == W2B_OK) st = encode_2d(enc, m, q, H.g, H.L, 32, (uint32_t)rows);
        };
        strip(&S.d, B.d, 1);
        strip(&S.qx, B.qx, 1);
        strip(&S.qy, B.qy, 2);
        strip(&S.zcx, B.zcx, 0);
        strip(&S.zcy, B.zcy, 1);
        for (int p = 0; p < 2; ++p) {
            strip(&S.h[p], B.h[p], 1);
            strip(&S.u[p], B.u[p], 4);
            strip(&S.v[p], B.v[p], 4);
            strip_own(&S.mx[p], B.mx[p]);
            strip_own(&S.my[p], B.my[p]);
        }
        // the resident loop's update of a strip: one row above to two below; its own rows of the residual and source
        UpdateMaps& U = H.rmaps[resident_index(rows)].u;
        strip(&U.qx1, B.qx1, 3);
        strip(&U.qy1, B.qy1, 3);
        for (int p = 0; p < 2; ++p) strip(&U.h[p], B.h[p], 3);
        strip_own(&U.res, B.res);
        strip_own(&U.src, B.src);
    }
    H.tmaps.s16 = H.rmaps[0].s;
    H.tmaps.s8 = H.rmaps[1].s;
    return st;
}

static void drop_graph(Handle& H, int c, int tail) {
    if (H.loop.exec[c][tail]) {
        cudaGraphExecDestroy(H.loop.exec[c][tail]);
        H.loop.exec[c][tail] = nullptr;
    }
    H.loop.version[c][tail] = ~0u;
}

static void drop_graph(Handle& H, int c) {
    for (int k = 0; k <= TAILS; ++k) drop_graph(H, c, k);
}

static void drop_graphs(Handle& H) {
    for (int c = 0; c <= TUNE_CANDIDATES; ++c) drop_graph(H, c);
}

// The tuner's candidates: the occupancy-given default (both passes at their resident CTAs a SM, 16 steps a graph), it
// with 32 steps a graph, the face pass in its strip forms, and the resident loop with each strip height.
static void init_loop(Handle& H) {
    Loop& L = H.loop;
    const int F = H.faces_occ, U = H.update_occ;
    auto fit = [&](int occ) { return occ < U ? occ : U; };
    L.ncand = 0;
    L.cand[L.ncand++] = {F, U, 16, 0, 0};
    L.cand[L.ncand++] = {F, U, 32, 0, 0};
    L.cand[L.ncand++] = {H.strips16_occ, U, 16, 16, 0};
    L.cand[L.ncand++] = {H.strips8_occ, U, 16, 8, 0};
    for (int i = 0; i < 3; ++i)
        L.cand[L.ncand++] = {H.resident_occ[i], fit(H.resident_occ[i]), 32, RESIDENT_ROWS[i], 1};
    L.cand[FORCED] = L.cand[0];
    for (int c = 0; c < TUNE_CANDIDATES; ++c) {
        L.sec[c] = 0.0;
        L.steps[c] = 0;
        L.samples[c] = 0;
    }
    L.next = L.chosen = 0;
    L.tuning = 1;
}

// CTAs of boundary_kernel: enough for its cells, at most four a SM.
static int boundary_grid(const Handle& H) {
    const int64_t g = (H.nb + 255) / 256;
    const int64_t cap = 4 * (int64_t)(H.sms > 0 ? H.sms : 148);
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// The shared-memory limits of both builds' passes, and the resident CTAs a SM of the handle's build (W2BParams.arith),
// which set the launch grids and the tuner's candidates.
static int set_passes(Handle& H) {
    for (const Passes* X : {&EXACT_PASSES, &FAST_PASSES}) {
        if (X->update_setup() != cudaSuccess || X->faces_setup() != cudaSuccess || X->resident_setup() != cudaSuccess)
            return cuda_status(cudaGetLastError(), "pass setup");
    }
    const Passes& X = passes(H.P);
    const int occ = X.update_occupancy(), focc = X.faces_occupancy();
    const int s16 = X.strips_occupancy(16), s8 = X.strips_occupancy(8);
    H.update_occ = occ > 0 ? occ : 1;
    H.faces_occ = focc > 0 ? focc : 1;
    H.strips16_occ = s16 > 0 ? s16 : 1;
    H.strips8_occ = s8 > 0 ? s8 : 1;
    for (int i = 0; i < 3; ++i) {
        const int occ = X.resident_occupancy(RESIDENT_ROWS[i]);
        H.resident_occ[i] = occ > 0 ? occ : 1;
    }
    H.step_blocks = H.sms * H.update_occ;
    H.faces_blocks = H.sms * H.faces_occ;
    init_loop(H);
    return W2B_OK;
}

// The pinned buffer: the run table, the control block, a batch's clocks and end times.
static size_t host_bytes(int nruns) {
    return run_table_bytes(nruns) + W2B_CTL_BYTES + (sizeof(W2BClock) + sizeof(double)) * (size_t)nruns;
}

// Before steps: the sleeping tiles' other halves, if a caller may have written their current ones.
static int settle_asleep(Handle& H, cudaStream_t s) {
    if (H.touched && H.B.is_act && H.nact < H.g.ntiles - 1) {
        launch_asleep(make_args(H), H.sms, s);
        CKL("sleeping tiles");
    }
    H.touched = false;
    return W2B_OK;
}

// The face pass of a host-driven step (w2b_step, w2b_step_timed) over n tiles: in the form and at the CTAs a SM the
// device loop's tuner settled on (strips of 8 rows for its resident loop of 8 or 4), and while it tunes in strips of 8
// rows, which are within 2 % of the fastest form of kernels of their own where a step is long (us, the tile form | 16 | 8
// rows, as w2b_step_timed has them: 1,645 tiles exact 107 | 93 | 95; 16,641 fast 638 | 570 | 564).
static void launch_faces_host(Handle& H, const StepArgs& A, int n, cudaStream_t s) {
    const LoopConfig& C = H.loop.cand[H.loop.chosen];
    const bool settled = !H.loop.tuning;
    if (settled && !C.strips) {
        passes(H.P).launch_faces(H.tmaps, A, faces_grid(H, n), s);
        return;
    }
    const int rows = settled && C.strips == 16 ? 16 : 8;
    const int occ = settled && !C.resident ? C.faces_per_sm : (rows == 16 ? H.strips16_occ : H.strips8_occ);
    const int g = H.sms * occ, units = (TILE / rows) * n;
    passes(H.P).launch_strips(rows, H.tmaps, A, units < g ? units : g, s);
}

// Step k of `steps` of a launch of the device loop under launch configuration C: every running run advances by one of its
// own steps. The steps take the two sets of settings in turn, the first step the first; the last leaves the next one's
// there.
static int launch_loop_step(Handle& H, const LoopConfig& C, int k, int steps, cudaStream_t s) {
    StepArgs A = make_args(H);
    A.list = A.work;
    if (k & 1) A = other_set(A);
    const int grid = blocks_for(H, H.g.ntiles - 1);
    const int tiles = H.g.ntiles - 1 > 0 ? H.g.ntiles - 1 : 1;
    const int fgrid = H.sms * C.faces_per_sm, ugrid = H.sms * C.update_per_sm;
    const Passes& X = passes(H.P);
    if (C.strips)
        X.launch_strips(C.strips, H.tmaps, A, (TILE / C.strips) * tiles < fgrid ? (TILE / C.strips) * tiles : fgrid, s);
    else
        X.launch_faces(H.tmaps, A, tiles < fgrid ? tiles : fgrid, s);
    X.launch_update(H.tmaps, A, (tiles < ugrid - 1 ? tiles : ugrid - 1) + 1, 1, s);
    // A step is five kernels; with the boundary cells, the clocks and settings as two more in a row it was 80 us instead of
    // 65 for ten catchments of 90 to 500 cells a side, 139 instead of 130 at 1500 x 1101, 865 instead of 840 at 4096^2.
    // the small kernels start while the one before them ends (grid_wait); the passes do not: CTAs that start as others
    // leave crowd onto the SMs that finish first, and the pass then waits for those (384 tiles: 57 us a step against 49)
    CK(launch_next(step_end_kernel, H.sms * 2, TILE2, 0, s, A));
    CK(launch_next(rebuild_kernel, 1, 1024, 0, s, A, k == steps - 1 && !(k & 1)));
    CK(launch_next(plan_kernel, grid, 256, 0, s, A, A.woken, -1));
    CKL("loop step");
    return W2B_OK;
}

// Cooperative launches on one device, whatever their streams: one may start beside others in flight only where all their
// CTAs are sure to find a place, for CTAs that wait at a grid barrier hold theirs until the last has come. A CTA of a kernel
// of which k are resident a SM takes at most 1 / k of everything a SM has, so a launch takes its CTAs / k SMs in all. While
// the launches in flight and this one take at most (1 - w) of the SMs together, w the largest 1 / k among them, some SM always
// has w of itself free, so every CTA finds room, in whatever order they come; with one k for all of them, a SM has room
// until it holds k CTAs, so they may take all the SMs. Else this launch waits, on the device, for the oldest ones. Calls of 20
// steps of eight models, a thread and a stream each: 328 us for all eight of 62 x 62 cells, 997 of 126 x 126 (two at a time),
// where 1,836 and 1,900 with every launch behind the one before it.
// A launch stands in the list, oldest first, under its stream (the stream's own order keeps it behind the ones before it on
// that), with what may run until it ends: what it takes, or what those it waits for take.
namespace {
struct Flight {
    unsigned long long stream;
    cudaEvent_t done;
    double sms, widest, narrowest;  // the SMs it takes; the largest and the smallest 1 / k
};
struct Lane {
    static constexpr int HELD = 16;
    std::mutex mutex;
    Flight held[HELD];
    cudaEvent_t spare[HELD] = {};
    int count = 0, spares = 0, sms = 0;
    void drop(int i) {
        spare[spares++] = held[i].done;
        for (--count; i < count; ++i) held[i] = held[i + 1];
    }
};
}  // namespace

cudaError_t launch_in_turn(const void* kernel, int grid, int block, void** params, size_t smem, int per_sm, cudaStream_t s) {
    static Lane lanes[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || per_sm < 1) return cudaErrorInvalidValue;
    Lane& L = lanes[dev];
    Flight mine = {0, nullptr, (double)grid / per_sm, 1.0 / per_sm, 1.0 / per_sm};
    e = cudaStreamGetId(s, &mine.stream);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(L.mutex);
    if (!L.sms) e = cudaDeviceGetAttribute(&L.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    double ahead = 0.0;  // SMs of launches that end before this one starts
    auto join = [](Flight& to, const Flight& f) {
        to.widest = f.widest > to.widest ? f.widest : to.widest;
        to.narrowest = f.narrowest < to.narrowest ? f.narrowest : to.narrowest;
    };
    auto behind = [&](int i) {
        ahead += L.held[i].sms;
        join(mine, L.held[i]);
        L.drop(i);
    };
    if (L.count > 1 || (L.count == 1 && L.held[0].stream != mine.stream)) {
        // the launches that have ended leave the list (a query would end another thread's capture in the default mode)
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        for (int i = L.count - 1; i >= 0; --i) {
            const cudaError_t ended = cudaEventQuery(L.held[i].done);
            if (ended == cudaSuccess) L.drop(i);
            if (ended == cudaErrorNotReady) cudaGetLastError();  // not an error to report
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    for (int i = L.count - 1; i >= 0; --i)
        if (L.held[i].stream == mine.stream) behind(i);
    auto fits = [&] {
        Flight all = mine;
        for (int i = 0; i < L.count; ++i) {
            all.sms += L.held[i].sms;
            join(all, L.held[i]);
        }
        return all.sms <= L.sms * (all.widest == all.narrowest ? 1.0 : 1.0 - all.widest);
    };
    while (L.count && (L.count == Lane::HELD || !fits())) {
        e = cudaStreamWaitEvent(s, L.held[0].done, 0);
        if (e != cudaSuccess) return e;
        behind(0);
    }
    mine.sms = mine.sms > ahead ? mine.sms : ahead;
    if (L.spares)
        mine.done = L.spare[--L.spares];
    else
        e = cudaEventCreateWithFlags(&mine.done, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
    e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(block), params, smem, s);
    const cudaError_t noted = cudaEventRecord(mine.done, s);  // (of a launch that failed too: it stands for those ahead)
    L.held[L.count++] = mine;
    return e != cudaSuccess ? e : noted;
}

// A launch of the resident loop over up to `tiles` tiles in strips of `rows` rows, at most per_sm CTAs a SM; where there is
// room, with CTAs of their own for the boundary cells, 32 each, whose loads then run beside the strips' (256 x 256 cells and
// 256 boundary cells, the envelope every fourth step: 16.7 us a step, 17.1 with all of them in one CTA).
static int launch_resident(Handle& H, const StepArgs& A, int rows, int per_sm, int64_t tiles, int max_steps,
                           const HostStep& host, cudaStream_t s) {
    const int64_t units = (int64_t)(TILE / rows) * tiles + (H.nb + 31) / 32;
    const int64_t most = (int64_t)H.sms * per_sm - 1;
    const int workers = (int)(units < most ? (units > 0 ? units : 1) : most);
    if (workers < 1) return W2B_EINVAL;
    const int form = resident_index(rows);
    CK(passes(H.P).launch_resident(rows, H.rmaps[form], A, workers + 1, H.resident_occ[form], max_steps, host, s));
    return W2B_OK;
}

// A host-driven step as one launch, where its strips of 8 rows are one wave of the resident kernel (then its two grid
// barriers cost less than the gaps between the passes' kernels: 81 tiles 18 us of GPU time against 27; at 384 tiles they
// are even) and the stream is not being captured (the launch waits for another stream's event). *done: whether it was.
static int host_resident(Handle& H, float dt, int want_wave, int want_wet, cudaStream_t s, bool* done) {
    *done = false;
    const int occ = H.resident_occ[resident_index(8)];
    if ((int64_t)(TILE / 8) * H.nact > (int64_t)H.sms * occ - 1) return W2B_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) return W2B_OK;
    if (want_wave) {
        CK(cudaMemsetAsync(H.B.wave, 0, sizeof(float) * H.g.ntiles, s));
        CK(cudaMemsetAsync(H.R.wave_bits, 0, sizeof(uint32_t), s));
    }
    StepArgs A = make_args(H);
    A.work = H.B.active;
    const HostStep host = {dt, F_RUN | (want_wave ? F_WAVE : 0) | (want_wet ? F_WET : 0), H.nact};
    *done = true;
    return launch_resident(H, A, 8, occ, H.nact, 1, host, s);
}

}  // namespace w2b

using namespace w2b;

extern "C" {

int32_t w2b_version(void) { return 3; }

int64_t w2b_run_table_bytes(int32_t nruns) { return nruns < 1 ? 0 : (int64_t)run_table_bytes(nruns); }

int32_t w2b_selftest_cbrt(uint32_t first_bits, uint32_t count, uint64_t* out, void* stream) {
    if (!out) return W2B_EINVAL;
    launch_cbrt_check(first_bits, count, reinterpret_cast<unsigned long long*>(out), (cudaStream_t)stream);
    CKL("w2b_selftest_cbrt");
    return W2B_OK;
}

int32_t w2b_selftest_wait(uint32_t polls, int64_t* out, void* stream) {
    if (!out || polls < 1 || polls > TMA_WAIT_LIMIT) return W2B_EINVAL;
    launch_wait_check(polls, reinterpret_cast<long long*>(out), (cudaStream_t)stream);
    CKL("w2b_selftest_wait");
    return W2B_OK;
}

int32_t w2b_layout(const W2BGridDesc* grid, W2BLayout* out) {
    if (!grid || !out || grid->ny <= 0 || grid->nx <= 0 || grid->ny % TILE || grid->nx % TILE || grid->ntiles < 1)
        return W2B_EINVAL;
    out->gy = GY;
    out->gx = GX;
    out->px = grid->nx + 2 * GX;
    out->ncells = (int64_t)(grid->ny + 2 * GY) * out->px;
    return W2B_OK;
}

int32_t w2b_ref_to_native(const W2BGridDesc* grid, const int32_t* tiles_host, int64_t n, const int64_t* ref_index,
                          int64_t* native_index) {
    W2BLayout L;
    if (w2b_layout(grid, &L) != W2B_OK || !tiles_host || n < 0 || (n && (!ref_index || !native_index)))
        return W2B_EINVAL;
    for (int64_t m = 0; m < n; ++m) {
        const int64_t k = ref_index[m];
        const int64_t t = k / 1296;
        if (k < 0 || t < 1 || t >= grid->ntiles) return W2B_EINVAL;
        const int64_t r = k % 1296;
        const int64_t j = (int64_t)tiles_host[2 * t] * TILE + r / 36 - 2;
        const int64_t i = (int64_t)tiles_host[2 * t + 1] * TILE + r % 36 - 2;
        native_index[m] = (j + L.gy) * L.px + i + L.gx;
    }
    return W2B_OK;
}

int32_t w2b_create(const W2BGridDesc* grid, const W2BParams* params, const W2BBuffers* buffers, void** handle) {
    if (!grid || !params || !buffers || !handle) return W2B_EINVAL;
    if (grid->rows < 4 || grid->rows > 64 || grid->nruns < 1) return W2B_EINVAL;
    if (params->arith != W2B_ARITH_EXACT && params->arith != W2B_ARITH_FAST) return W2B_EINVAL;
    if (!buffers->runs || ((uintptr_t)buffers->runs & 255) || !buffers->tile_run || !buffers->work) return W2B_EINVAL;
    {
        // arrays the passes stage with bulk copies: 16-byte aligned
        auto a16 = [](const void* q) { return q && !((uintptr_t)q & 15); };
        bool ok = a16(buffers->hc) && a16(buffers->lpair) && a16(buffers->lrow);
        for (int x = 0; x < 2; ++x)
            ok = ok && a16(buffers->fl[x]) && a16(buffers->fr[x]) && a16(buffers->gl[x]) && a16(buffers->gr[x]) &&
                 a16(buffers->ef[x]) && a16(buffers->cw[x]);
        for (int e = 0; e < 5; ++e) ok = ok && a16(buffers->env[e]);
        if (!ok) return W2B_EINVAL;
    }
    Handle* H = new (std::nothrow) Handle();
    if (!H) return W2B_EINVAL;
    H->g = *grid;
    H->P = *params;
    H->B = *buffers;
    if (w2b_layout(grid, &H->L) != W2B_OK || !H->B.ctl || ((uintptr_t)H->B.ctl & 255)) {
        delete H;
        return W2B_EINVAL;
    }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&H->sms, cudaDevAttrMultiProcessorCount, dev);
    if (set_passes(*H) != W2B_OK) {
        delete H;
        return W2B_ECUDA;
    }
    if (build_tmaps(*H) != W2B_OK) {
        delete H;
        return W2B_ECUDA;
    }
    H->nact = grid->ntiles - 1;
    H->nruns = grid->nruns;
    H->R = run_table(H->B.runs, H->nruns);
    // the level cache holds nothing yet: every row 0xff
    if (cudaMemset(H->B.lrow, 0xff, (size_t)H->g.ntiles * TILE2) != cudaSuccess) {
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create level cache");
    }
    const int32_t stored = 1;  // the caller's momentum arrays hold the momenta the first step starts from
    if (cudaMemcpy(&H->ctl()->m_stored, &stored, sizeof(stored), cudaMemcpyHostToDevice) != cudaSuccess) {
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create control block");
    }
    if (cudaMemset(reinterpret_cast<char*>(H->ctl()) + GRID_STATE_AT, 0, sizeof(GridState)) != cudaSuccess) {
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create grid state");
    }
    if (H->nruns == 1 && cudaMemcpy(H->R.dx, &H->P.dx, sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) {
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create run table");
    }
    if (cudaMallocHost(&H->host, host_bytes(H->nruns)) != cudaSuccess) {
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create read-back");
    }
    if (cudaStreamCreateWithFlags(&H->cap, cudaStreamNonBlocking) != cudaSuccess) {
        cudaFreeHost(H->host);
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create stream");
    }
    if (cudaEventCreate(&H->loop.ev[0]) != cudaSuccess || cudaEventCreate(&H->loop.ev[1]) != cudaSuccess ||
        cudaEventCreate(&H->loop.ev[2]) != cudaSuccess) {
        for (auto& e : H->loop.ev)
            if (e) cudaEventDestroy(e);
        cudaStreamDestroy(H->cap);
        cudaFreeHost(H->host);
        delete H;
        return cuda_status(cudaGetLastError(), "w2b_create events");
    }
    const int st = cuda_status(cudaGetLastError(), "w2b_create");
    if (st != W2B_OK) {  // no handle goes out with a failure: the caller has nothing to destroy
        w2b_destroy(H);
        return st;
    }
    *handle = H;
    return W2B_OK;
}

int32_t w2b_destroy(void* handle) {
    if (!handle) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    drop_graphs(*H);
    for (auto& e : H->loop.ev)
        if (e) cudaEventDestroy(e);
    if (H->cap) cudaStreamDestroy(H->cap);
    if (H->host) cudaFreeHost(H->host);
    delete H;
    return W2B_OK;
}

int32_t w2b_pack_tables(const W2BGridDesc* grid, const float* dtab, const float* ftabx, const float* ftaby,
                        float* dtab2, float* ftab4x, float* ftab4y, void* stream) {
    if (!grid || !dtab || !ftabx || !ftaby || !dtab2 || !ftab4x || !ftab4y || grid->rows < 4) return W2B_EINVAL;
    if (((uintptr_t)dtab2 & 7) || ((uintptr_t)ftab4x & 15) || ((uintptr_t)ftab4y & 15)) return W2B_EINVAL;
    pack_tables_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(dtab, ftabx, ftaby, reinterpret_cast<float2*>(dtab2),
                                                              reinterpret_cast<float4*>(ftab4x),
                                                              reinterpret_cast<float4*>(ftab4y), grid->ntiles,
                                                              grid->rows);
    CKL("w2b_pack_tables");
    return W2B_OK;
}

int32_t w2b_set_params(void* handle, const W2BParams* params) {
    if (!handle || !params) return W2B_EINVAL;
    if (params->arith != W2B_ARITH_EXACT && params->arith != W2B_ARITH_FAST) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    const int arith = H->P.arith;
    H->P = *params;
    H->version++;
    if (params->arith != arith) {  // the other build's passes: their occupancy, and the tuner starts again
        drop_graphs(*H);
        const int st = set_passes(*H);
        if (st != W2B_OK) return st;
    }
    if (H->nruns == 1) CK(cudaMemcpy(H->R.dx, &H->P.dx, sizeof(float), cudaMemcpyHostToDevice));
    return W2B_OK;
}

int32_t w2b_set_active(void* handle, const int32_t* tiles, int32_t n, void* stream) {
    if (!handle || n < 0) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (n > H->g.ntiles - 1 || (n && !tiles)) return W2B_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    if (n && tiles != H->B.active)
        CK(cudaMemcpyAsync(H->B.active, tiles, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
    H->nact = n;
    if (H->B.is_act) active_flags_kernel<<<1, 1024, 0, s>>>(make_args(*H), n);
    CKL("w2b_set_active");
    return W2B_OK;
}

int32_t w2b_set_boundary(void* handle, int32_t n, const int32_t* cell, const int32_t* ref, const int32_t* kind,
                         const float* d0, const float* h0) {
    if (!handle || n < 0 || (n && (!cell || !ref || !kind || !d0 || !h0))) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    H->nb = n;
    H->bcell = cell;
    H->bref = ref;
    H->bkind = kind;
    H->bd0 = d0;
    H->bh0 = h0;
    H->version++;
    const StepArgs A = make_args(*H);
    bmark_kernel<<<64, 256>>>(A, H->g.ntiles * TILE);
    if (n) bmark_kernel<<<64, 256>>>(A, 0);
    CKL("w2b_set_boundary");
    return W2B_OK;
}

int32_t w2b_set_tally(void* handle, int32_t n, const int32_t* face, const int32_t* axis, const float* sign,
                      double* total) {
    if (!handle || n < 0 || (n && (!face || !axis || !sign || !total))) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    H->ntally = n;
    H->tface = face;
    H->taxis = axis;
    H->tsign = sign;
    H->ttotal = total;
    H->version++;
    return W2B_OK;
}

int32_t w2b_set_lines(void* handle, int32_t nlines, const int32_t* start, const int32_t* face, const int32_t* axis,
                      const float* sign, double* q, double* peak, double* time) {
    if (!handle || nlines < 0 || (nlines && (!start || !face || !axis || !sign || !q || !peak || !time)))
        return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    H->nlines = nlines;
    H->lstart = start;
    H->lface = face;
    H->laxis = axis;
    H->lsign = sign;
    H->lq = q;
    H->lpeak = peak;
    H->ltime = time;
    H->version++;
    return W2B_OK;
}

int32_t w2b_step(void* handle, float dt, int32_t want_wave, int32_t want_wet, void* stream) {
    if (!handle) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    cudaStream_t s = (cudaStream_t)stream;
    if (H->nruns != 1) return W2B_EINVAL;  // a batch steps in the device loop
    if (H->nact > 0) {
        bool done = false;
        int st = settle_asleep(*H, s);
        if (st == W2B_OK) st = host_resident(*H, dt, want_wave, want_wet, s, &done);
        if (st != W2B_OK) return st;
        if (done) {
            H->cur ^= 1;
            return W2B_OK;
        }
    }
    const StepArgs A = make_args(*H);
    setstep_kernel<<<1, want_wave ? 1024 : 32, 0, s>>>(A, dt, want_wave, want_wet, H->nact);
    if (H->nact == 0) {  // as the reference: no tiles, no swap
        CKL("w2b_step");
        return W2B_OK;
    }
    const int grid = blocks_for(*H, H->nact);
    launch_faces_host(*H, A, H->nact, s);
    passes(H->P).launch_update(H->tmaps, A, grid, 0, s);
    CK(launch_next(boundary_kernel, boundary_grid(*H), 256, 0, s, A));
    CKL("w2b_step");
    H->cur ^= 1;
    return W2B_OK;
}

int32_t w2b_step_timed(void* handle, float dt, int32_t want_wave, int32_t want_wet, void* stream, float* ms) {
    if (!handle || !ms) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    cudaStream_t s = (cudaStream_t)stream;
    if (H->nact == 0 || H->nruns != 1) return W2B_EINVAL;
    const int st = settle_asleep(*H, s);
    if (st != W2B_OK) return st;
    cudaEvent_t ev[4];
    for (auto& e : ev) CK(cudaEventCreate(&e));
    const StepArgs A = make_args(*H);
    setstep_kernel<<<1, 1024, 0, s>>>(A, dt, want_wave, want_wet, H->nact);
    const int grid = blocks_for(*H, H->nact);
    CK(cudaEventRecord(ev[0], s));
    launch_faces_host(*H, A, H->nact, s);
    CK(cudaEventRecord(ev[1], s));
    passes(H->P).launch_update(H->tmaps, A, grid, 0, s);
    CK(cudaEventRecord(ev[2], s));
    boundary_kernel<<<boundary_grid(*H), 256, 0, s>>>(A);
    CK(cudaEventRecord(ev[3], s));
    CKL("w2b_step_timed");
    H->cur ^= 1;
    CK(cudaEventSynchronize(ev[3]));
    for (int e = 0; e < 3; ++e) CK(cudaEventElapsedTime(ms + e, ev[e], ev[e + 1]));
    for (auto& e : ev) cudaEventDestroy(e);
    return W2B_OK;
}

int32_t w2b_max_wave(void* handle, float* out, void* stream) {
    if (!handle || !out) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    int32_t* const held = reinterpret_cast<int32_t*>(H->host);  // pinned: the two copies queue without the host
    CK(cudaMemcpyAsync(held, H->R.wave_bits, sizeof(float), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    CK(cudaMemcpyAsync(held + 1, &H->ctl()->status, sizeof(int32_t), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    CK(cudaStreamSynchronize((cudaStream_t)stream));
    memcpy(out, held, sizeof(float));
    if (held[1] != W2B_ETIMEOUT) return W2B_OK;
    // the device's half: a step that gave up, and one that a failure kept from beginning, swapped nothing there
    CK(cudaMemcpyAsync(held, H->R.parity, sizeof(int32_t), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    CK(cudaStreamSynchronize((cudaStream_t)stream));
    H->cur = held[0];
    return W2B_ETIMEOUT;
}

int32_t w2b_wet_flags(void* handle, int32_t* out, void* stream) {
    if (!handle || !out) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    CK(cudaMemcpyAsync(out, H->B.wet, sizeof(int32_t) * H->g.ntiles, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    CK(cudaStreamSynchronize((cudaStream_t)stream));
    return W2B_OK;
}

int32_t w2b_refresh_plan(void* handle, const int32_t* tiles, int32_t n, void* stream) {
    if (!handle || n < 0 || (n && !tiles)) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (!n) return W2B_OK;
    const StepArgs A = make_args(*H);
    plan_kernel<<<blocks_for(*H, n), 256, 0, (cudaStream_t)stream>>>(A, tiles, n);
    CKL("w2b_refresh_plan");
    return W2B_OK;
}

static float* field_ptr(Handle* H, int f) {
    const int c = H->cur, o = 1 - H->cur;
    switch (f) {
        case W2B_H: return H->B.h[c];
        case W2B_D: return H->B.d;
        case W2B_U: return H->B.u[c];
        case W2B_V: return H->B.v[c];
        case W2B_MX: return H->B.mx[c];
        case W2B_MY: return H->B.my[c];
        case W2B_QX: return H->B.qx;
        case W2B_QY: return H->B.qy;
        case W2B_U1: return H->B.u[o];
        case W2B_V1: return H->B.v[o];
        case W2B_MX1: return H->B.mx[o];
        case W2B_MY1: return H->B.my[o];
        case W2B_QX1: return H->B.qx1;
        case W2B_QY1: return H->B.qy1;
        case W2B_SRC: return H->B.src;
        case W2B_RES: return H->B.res;
        case W2B_OM: return H->B.om;
        case W2B_ZCX: return H->B.zcx;
        case W2B_ZCY: return H->B.zcy;
        default: return nullptr;
    }
}

int32_t w2b_cell_size(void* handle, float* dx) {
    if (!handle || !dx) return W2B_EINVAL;
    *dx = static_cast<Handle*>(handle)->P.dx;
    return W2B_OK;
}

int32_t w2b_field_read(void* handle, int32_t field, const float** out) {
    if (!handle || !out) return W2B_EINVAL;
    const float* p = field_ptr(static_cast<Handle*>(handle), field);
    if (!p) return W2B_EINVAL;
    *out = p;
    return W2B_OK;
}

int32_t w2b_field_ptr(void* handle, int32_t field, float** out) {
    if (!handle || !out) return W2B_EINVAL;
    const float* p = nullptr;
    const int st = w2b_field_read(handle, field, &p);
    if (st != W2B_OK) return st;
    *out = const_cast<float*>(p);
    if (field == W2B_H || field == W2B_U || field == W2B_V) static_cast<Handle*>(handle)->touched = true;
    return W2B_OK;
}

// Fields whose reading or writing needs the momenta in their arrays: the momenta themselves, and the velocities they
// are formed from (a velocity written afterwards must not change the momentum the next step starts from).
static bool momentum_field(int f) {
    return f == W2B_U || f == W2B_V || f == W2B_MX || f == W2B_MY || f == W2B_U1 || f == W2B_V1 || f == W2B_MX1 ||
           f == W2B_MY1;
}

static int sync_momentum(Handle& H, cudaStream_t s) {
    launch_momentum(make_args(H), H.sms, s);
    CKL("w2b_sync_momentum");
    return W2B_OK;
}

int32_t w2b_get_field(void* handle, int32_t field, float* dst, int32_t layout, int32_t host, void* stream) {
    if (!handle || !dst) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    float* src = field_ptr(H, field);
    if (!src) return W2B_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    if (momentum_field(field)) {
        const int st = sync_momentum(*H, s);
        if (st != W2B_OK) return st;
    }
    if (layout == W2B_LAYOUT_NATIVE) {
        CK(cudaMemcpyAsync(dst, src, sizeof(float) * H->L.ncells,
                           host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, s));
    } else if (layout == W2B_LAYOUT_REF_TILE) {
        float* out = host ? H->B.stage : dst;
        native_to_ref_kernel<<<H->g.ntiles, 256, 0, s>>>(src, out, H->B.tiles, H->B.tile_of, H->g.ntiles, H->g.ny,
                                                         H->g.nx, H->L.px);
        CKL("native_to_ref");
        if (host)
            CK(cudaMemcpyAsync(dst, out, sizeof(float) * 1296 * (size_t)H->g.ntiles, cudaMemcpyDeviceToHost, s));
    } else {
        return W2B_EINVAL;
    }
    if (host) CK(cudaStreamSynchronize(s));
    return W2B_OK;
}

int32_t w2b_set_field(void* handle, int32_t field, const float* src, int32_t layout, int32_t host, void* stream) {
    if (!handle || !src) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    float* dst = field_ptr(H, field);
    if (!dst) return W2B_EINVAL;
    if (field == W2B_H || field == W2B_U || field == W2B_V) H->touched = true;
    cudaStream_t s = (cudaStream_t)stream;
    if (momentum_field(field)) {
        const int st = sync_momentum(*H, s);
        if (st != W2B_OK) return st;
    }
    if (layout == W2B_LAYOUT_NATIVE) {
        CK(cudaMemcpyAsync(dst, src, sizeof(float) * H->L.ncells,
                           host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, s));
    } else if (layout == W2B_LAYOUT_REF_TILE) {
        const float* in = src;
        if (host) {
            CK(cudaMemcpyAsync(H->B.stage, src, sizeof(float) * 1296 * (size_t)H->g.ntiles, cudaMemcpyHostToDevice,
                               s));
            in = H->B.stage;
        }
        ref_to_native_kernel<<<H->g.ntiles - 1 > 0 ? H->g.ntiles - 1 : 1, 256, 0, s>>>(in, dst, H->B.tiles,
                                                                                       H->g.ntiles, H->L.px);
        CKL("ref_to_native");
    } else {
        return W2B_EINVAL;
    }
    if (host) CK(cudaStreamSynchronize(s));
    return W2B_OK;
}

int32_t w2b_sync_momentum(void* handle, void* stream) {
    if (!handle) return W2B_EINVAL;
    return sync_momentum(*static_cast<Handle*>(handle), (cudaStream_t)stream);
}

int32_t w2b_maxima(void* handle, float t, float arrive, float deep, void* stream) {
    if (!handle) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (!H->nact) return W2B_OK;
    const StepArgs A = make_args(*H);
    maxima_kernel<<<blocks_for(*H, H->nact), dim3(32, 8), 0, (cudaStream_t)stream>>>(A, t, arrive, deep, H->nact);
    CKL("w2b_maxima");
    return W2B_OK;
}

int32_t w2b_tally(void* handle, double dt, void* stream) {
    if (!handle) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (!H->ntally) return W2B_OK;
    const StepArgs A = make_args(*H);
    tally_kernel<<<(H->ntally + 255) / 256, 256, 0, (cudaStream_t)stream>>>(A, dt);
    CKL("w2b_tally");
    return W2B_OK;
}

// The graph of configuration c, of its steps (tail 0) or of TAIL_STEPS[tail - 1], captured again when the arguments it
// would hold have changed.
static int loop_graph(Handle& H, int c, int tail) {
    Loop& L = H.loop;
    if (L.exec[c][tail] && L.version[c][tail] == H.version) return W2B_OK;
    drop_graph(H, c, tail);
    cudaGraph_t graph;
    CK(cudaStreamBeginCapture(H.cap, cudaStreamCaptureModeThreadLocal));
    int stc = W2B_OK;
    const int steps = tail ? TAIL_STEPS[tail - 1] : L.cand[c].steps;
    for (int k = 0; k < steps && stc == W2B_OK; ++k) stc = launch_loop_step(H, L.cand[c], k, steps, H.cap);
    cudaError_t e = cudaStreamEndCapture(H.cap, &graph);
    if (stc != W2B_OK) {
        if (e == cudaSuccess) cudaGraphDestroy(graph);
        return stc;
    }
    CK(e);
    e = cudaGraphInstantiate(&L.exec[c][tail], graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) L.exec[c][tail] = nullptr;  // nothing to destroy later
    CK(e);
    L.version[c][tail] = H.version;
    return W2B_OK;
}

// One launch of `steps` loop steps of configuration c, or of fewer: the resident loop stops by itself, and a graph of
// the configuration's steps is made up of whole ones and of tails. Returns the status; *took: the steps launched.
static int launch_chunk(Handle& H, int c, int64_t steps, int64_t* took, cudaStream_t s) {
    Loop& L = H.loop;
    const LoopConfig& C = L.cand[c];
    *took = C.steps;
    if (C.resident)
        return launch_resident(H, make_args(H), C.strips, C.faces_per_sm, H.g.ntiles - 1, C.steps, HostStep{}, s);
    int tail = 0;
    while (tail < TAILS && *took > steps) *took = TAIL_STEPS[tail++];
    const int st = loop_graph(H, c, tail);
    if (st != W2B_OK) return st;
    CK(cudaGraphLaunch(L.exec[c][tail], s));
    return W2B_OK;
}

// Whether the tuner tries candidate k on `nact` active tiles: the resident loop only up to two waves of its strips. Beyond
// them its launches cost more than the step's kernels everywhere measured, all cells wet, exact (us a step, kernels | 16- | 8-
// | 4-row strips; waves in brackets): 121 tiles 22.9 | 19.3 (0.8) | 25.5 (1.1) | 25.8 (3.3); 196 26.1 | 30.5 (1.3) | 26.0
// (1.8) | 35.1 (5.3); 256 28.8 | 31.0 (1.7) | 35.1 (2.3) | 41.2; 484 44.5 | 56.2 (3.3) | 54.1 (4.4) | 77.6; 1,645 112 | 161 |
// 150 | 250. At 4096 x 4096 trying them made the first 900 steps of a handle 842 ms instead of 650.
static bool tried(const Handle& H, int k, int64_t nact) {
    const LoopConfig& C = H.loop.cand[k];
    return !C.resident || (int64_t)(TILE / C.strips) * nact <= 2 * ((int64_t)H.sms * C.faces_per_sm - 1);
}

// The candidate that the tuner times next.
static int next_candidate(const Handle& H, int64_t nact) {
    const Loop& L = H.loop;
    int c = L.next;
    while (!tried(H, c, nact)) c = (c + 1) % L.ncand;  // (the first candidates are not resident)
    return c;
}

// One timed launch of candidate c ran `live` loop steps in `ms`: add it, move to the next candidate, and settle on the
// fastest once every candidate that is tried on `nact` tiles has its samples; then with the graphs of fewer steps that it will take, so that the first
// call to end in one does not pay for them (222 us of a call of 13 steps of 484 tiles, which takes 663).
static int tune_sample(Handle& H, int c, int64_t nact, long long live, float ms, cudaStream_t s) {
    Loop& L = H.loop;
    if (live > 0) {
        L.sec[c] += 1e-3 * (double)ms;
        L.steps[c] += live;
        L.samples[c] += 1;
    }
    L.next = (c + 1) % L.ncand;
    for (int k = 0; k < L.ncand; ++k)
        if (tried(H, k, nact) && L.samples[k] < TUNE_SAMPLES) return W2B_OK;
    auto per_step = [&](int k) { return L.sec[k] / (double)(L.steps[k] > 0 ? L.steps[k] : 1); };
    int best = 0;
    for (int k = 1; k < L.ncand; ++k)
        if (tried(H, k, nact) && per_step(k) < per_step(best)) best = k;
    if (best != 0 && !(per_step(best) < (1.0 - TUNE_MARGIN) * per_step(0))) best = 0;
    L.chosen = best;
    L.tuning = 0;
    for (int k = 0; k < L.ncand; ++k)
        if (k != best) drop_graph(H, k);
    int st = W2B_OK;
    for (int tail = 1; tail <= TAILS && st == W2B_OK && !L.cand[best].resident; ++tail) {
        st = loop_graph(H, best, tail);
        if (st == W2B_OK) st = cuda_status(cudaGraphUpload(L.exec[best][tail], s), "cudaGraphUpload");
    }
    return st;
}

// The device-resident loop. Steps run in chunks (a captured graph, or one launch of the resident loop), every running
// run advancing one of its own steps each loop step; after a few chunks the host reads the run table and the control
// block once, into pinned memory. Empty steps at the end of a call cost a launch of every kernel each (about 20 us for
// 1,680 tiles), so the last chunks are graphs of fewer steps.
constexpr int CHUNKS = 8;
static int advance_runs(Handle* H, const W2BStepper* cfg, const double* t_end, int64_t max_steps, W2BClock* clocks,
                        cudaStream_t s) {
    const int n = H->nruns;
    Ctl c;
    memset(&c, 0, sizeof(c));
    c.nact = H->nact;
    c.nruns = n;
    c.dt_every = cfg->dt_every;
    c.active_every = cfg->active_every;
    c.adaptive = cfg->adaptive;
    c.max_every = cfg->max_every;
    c.arrive = cfg->arrive;
    c.deep = cfg->deep;
    c.cfl = cfg->cfl;
    c.wave_floor = cfg->wave_floor;
    c.dt_max = cfg->dt_max;
    c.dt_min = cfg->dt_min;
    // A single run's settings and clock travel as kernel arguments: a copy from the host would be queued on a copy
    // engine behind any large upload in flight on another stream (the next window's source, staged while this window
    // steps) and wait for it. A batch's are read from the pinned buffer by the kernel itself.
    char* const held = H->host;
    Ctl* const hctl = reinterpret_cast<Ctl*>(held + run_table_bytes(n));
    W2BClock* const hclocks = reinterpret_cast<W2BClock*>(held + run_table_bytes(n) + W2B_CTL_BYTES);
    double* const hends = reinterpret_cast<double*>(hclocks + n);
    if (n > 1) {
        memcpy(hclocks, clocks, sizeof(W2BClock) * n);
        memcpy(hends, t_end, sizeof(double) * n);
    }
    const int settled = settle_asleep(*H, s);
    if (settled != W2B_OK) return settled;
    // the work list of the runs that take a step, and the first step's settings; each step sets the next's
    begin_kernel<<<1, 1024, 0, s>>>(make_args(*H), c, clocks[0], t_end[0], (long long)max_steps,
                                    n > 1 ? hclocks : nullptr, n > 1 ? hends : nullptr);
    CKL("advance begin");
    const RunTab T = run_table(held, n);
    Loop& L = H->loop;
    int64_t nact = H->nact;
    long long ran_before = 0;  // loop steps so far in this call (the largest steps_run of any run)
    bool first_round = true;     // the runs' clocks are the caller's, not yet read back
    int end = 1, have_prev = 0;  // ev[end] takes this launch's end; ev[3 - end] holds the last one's, if have_prev
    if (L.tuning)  // every candidate's graph before the first timed launch: no capture falls inside a timing
        for (int k = 0; k < L.ncand; ++k) {
            const int stc = L.cand[k].resident ? W2B_OK : loop_graph(*H, k, 0);
            if (stc != W2B_OK) return stc;
        }
    for (;;) {
        const bool timed = L.tuning != 0;
        const int c = timed ? next_candidate(*H, nact) : L.chosen;
        if (timed && !have_prev) CK(cudaEventRecord(L.ev[0], s));
        // a timed launch is one of the candidate's steps; else as many as the runs will want at their current steps (a
        // step rule that shortens them on the way takes another round), at most CHUNKS before the host looks
        int64_t want = L.cand[c].steps;
        if (!timed) {
            want = 1;
            for (int r = 0; r < n; ++r) {
                double dt = first_round ? clocks[r].dt : T.dt[r];
                dt = dt < cfg->dt_max ? dt : cfg->dt_max;
                const double left = t_end[r] - (first_round ? clocks[r].t : T.t[r]);
                const int64_t cap = max_steps - (first_round ? 0 : T.steps_run[r]);
                const double est = dt > 0.0 ? ceil((left - 1e-9) / dt) : 1.0;
                const int64_t need = est < (double)cap ? (int64_t)est : cap;
                if ((first_round || T.status[r] == 0) && need > want) want = need;
            }
        }
        first_round = false;
        for (int k = 0; k < (timed ? 1 : CHUNKS) && want > 0; ++k) {
            int64_t took = 0;
            const int stc = launch_chunk(*H, c, want, &took, s);
            if (stc != W2B_OK) return stc;
            want -= took;
        }
        if (timed) CK(cudaEventRecord(L.ev[end], s));
        CK(cudaMemcpyAsync(held, H->B.runs, run_table_bytes(n), cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(hctl, H->ctl(), sizeof(Ctl), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        nact = hctl->nact;
        if (timed) {
            long long ran = 0;
            for (int r = 0; r < n; ++r) ran = T.steps_run[r] > ran ? T.steps_run[r] : ran;
            float ms = 0.0f;
            CK(cudaEventElapsedTime(&ms, have_prev ? L.ev[3 - end] : L.ev[0], L.ev[end]));
            const int stc = tune_sample(*H, c, nact, ran - ran_before, ms, s);
            if (stc != W2B_OK) return stc;
            ran_before = ran;
            have_prev = 1;
            end = 3 - end;
        } else {
            have_prev = 0;
        }
        bool done = hctl->status != 0;
        if (!done) {
            done = true;
            for (int r = 0; r < n; ++r)
                if (T.status[r] == 0 && T.t[r] < t_end[r] - 1e-9 && T.steps_run[r] < max_steps) done = false;
        }
        if (done) break;
    }
    const int32_t gstatus = hctl->status;
    H->nact = hctl->nact;
    H->cur = T.parity[0];
    int32_t first = gstatus;
    for (int r = 0; r < n; ++r) {
        clocks[r].t = T.t[r];
        clocks[r].dt = T.dt[r];
        clocks[r].nsteps = T.nsteps[r];
        clocks[r].refresh_due = 0;
        clocks[r].status = T.status[r] != 0 ? T.status[r] : gstatus;
        clocks[r].wave_max = T.wave_last[r];
        clocks[r].nact = hctl->nact;
        if (!first && T.status[r]) first = T.status[r];
    }
    return first;
}

int32_t w2b_advance(void* handle, const W2BStepper* cfg, double t_end, int64_t max_steps, W2BClock* clock,
                    void* stream) {
    if (!handle || !cfg || !clock || max_steps < 0 || cfg->dt_every < 1 || cfg->active_every < 1) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (H->nruns != 1) return W2B_EINVAL;
    return advance_runs(H, cfg, &t_end, max_steps, clock, (cudaStream_t)stream);
}

int32_t w2b_advance_runs(void* handle, const W2BStepper* cfg, const double* t_end, int64_t max_steps,
                         W2BClock* clocks, void* stream) {
    if (!handle || !cfg || !clocks || !t_end || max_steps < 0 || cfg->dt_every < 1 || cfg->active_every < 1)
        return W2B_EINVAL;
    return advance_runs(static_cast<Handle*>(handle), cfg, t_end, max_steps, clocks, (cudaStream_t)stream);
}

int32_t w2b_loop_tuning(void* handle, int32_t tune, int32_t faces_per_sm, int32_t update_per_sm, int32_t steps) {
    if (!handle) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    Loop& L = H->loop;
    if (tune == 1) {
        drop_graphs(*H);
        init_loop(*H);
        return W2B_OK;
    }
    if (tune < 0 || tune > 6) return W2B_EINVAL;
    const int resident = tune >= 4, strips = resident ? RESIDENT_ROWS[tune - 4] : (tune == 2 ? 16 : (tune == 3 ? 8 : 0));
    const int occ = resident ? H->resident_occ[tune - 4]
                             : (strips == 16 ? H->strips16_occ : (strips == 8 ? H->strips8_occ : H->faces_occ));
    if (faces_per_sm < 1 || faces_per_sm > occ || update_per_sm < 1 ||
        update_per_sm > H->update_occ || steps < 1 || steps > MAX_GRAPH_STEPS)
        return W2B_EINVAL;
    L.cand[FORCED] = {faces_per_sm, update_per_sm, steps, strips, resident};
    drop_graph(*H, FORCED);
    L.chosen = FORCED;
    L.tuning = 0;
    return W2B_OK;
}

int32_t w2b_loop_config(void* handle, int32_t* out) {
    if (!handle || !out) return W2B_EINVAL;
    const Handle* H = static_cast<const Handle*>(handle);
    const Loop& L = H->loop;
    const LoopConfig& C = L.cand[L.tuning ? next_candidate(*H, H->nact) : L.chosen];
    out[0] = C.faces_per_sm;
    out[1] = C.update_per_sm;
    out[2] = C.steps;
    out[3] = L.tuning;
    out[4] = H->faces_occ;
    out[5] = H->update_occ;
    out[6] = C.strips;
    out[7] = H->strips16_occ;
    out[8] = H->strips8_occ;
    return W2B_OK;
}

int32_t w2b_loop_resident(void* handle, int32_t* out) {
    if (!handle || !out) return W2B_EINVAL;
    const Handle* H = static_cast<const Handle*>(handle);
    const Loop& L = H->loop;
    out[0] = L.cand[L.tuning ? next_candidate(*H, H->nact) : L.chosen].resident;
    for (int i = 0; i < 3; ++i) out[1 + i] = H->resident_occ[i];
    return W2B_OK;
}

int32_t w2b_face_waves(void* handle, int32_t tile, float dt, float* out, void* stream) {
    if (!handle || !out || !(dt > 0.0f)) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (tile < 1 || tile >= H->g.ntiles) return W2B_EINVAL;
    passes(H->P).launch_probe(make_args(*H), tile, dt, out, (cudaStream_t)stream);
    CKL("w2b_face_waves");
    return W2B_OK;
}

int32_t w2b_run_halves(void* handle, int32_t* out, void* stream) {
    if (!handle || !out) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaMemcpyAsync(out, H->R.parity, sizeof(int32_t) * H->nruns, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return W2B_OK;
}

int32_t w2b_set_run_dx(void* handle, const float* dx, int32_t n) {
    if (!handle || !dx) return W2B_EINVAL;
    Handle* H = static_cast<Handle*>(handle);
    if (n != H->nruns) return W2B_EINVAL;
    CK(cudaMemcpy(H->R.dx, dx, sizeof(float) * n, cudaMemcpyHostToDevice));
    return W2B_OK;
}

}  // extern "C"
