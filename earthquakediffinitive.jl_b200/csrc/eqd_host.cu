// libeqd host side: grid set-up, launch geometry, the batched CG driver and
// the C ABI declared in include/eqd.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <condition_variable>
#include <deque>
#include <map>
#include <string>
#include <thread>
#include <vector>

#include "../../include/eqd.h"
#include "ops_tables.h"
#include "solver_kernels.cuh"
#include "rhs_kernels.cuh"
#include "ring_march.cuh"
#include "resident_cg.cuh"
#include "xmarch.cuh"

using namespace eqd;

// ---------------------------------------------------------------------------
// Errors
// ---------------------------------------------------------------------------
static thread_local std::string g_last_error;

static int fail(int code, const std::string &msg) {
    g_last_error = msg;
    return code;
}

#define CUDA_OR_RETURN(call)                                                                       \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            return fail(e_ == cudaErrorMemoryAllocation ? EQD_ERR_OOM : EQD_ERR_CUDA,              \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                       \
        }                                                                                          \
    } while (0)

// ---------------------------------------------------------------------------
// Device buffers
// ---------------------------------------------------------------------------
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        release();
        cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) bytes = n;
        else p = nullptr;
        return e;
    }
    template <typename T> T *as() const { return static_cast<T *>(p); }
};

// Launch configuration of the plane-march apply for one precision.
struct MarchCfg {
    MarchGeom g;
    int threads = 0;
    size_t smem = 0;
    size_t smem_af = 0;  // MODE_AF (second plane ring); 0: does not fit, the direction update runs apart
    int ring_t2 = 0;     // > 0: the FP32 A-apply runs ring_march_kernel with this x2 tile capacity
    int ring_var = 0;    // which of the two ring-march instances of this n1 (0: A, 1: B)
    RingGeom rg{};
};

static constexpr int kMaxT32 = 640;   // generic FP32 instances
static constexpr int kMaxT32b = 512;  // FP32 A-apply variant without register spills
static constexpr int kMaxT32c = 384;  // FP32 A-apply, two columns per thread
static constexpr int kMaxT64 = 384;
static constexpr int kMaxT64b = 512;  // FP64 instances for wide x1 lines (n1 = 33 needs 7 x 66 threads)
static constexpr int kNumVariants = 11;  // 9 plane-march variants, then 2 ring-march variants
static constexpr int kFirstRingVariant = 9;
static constexpr int kResidentVariant = kNumVariants;  // whole iterations resident on chip (resident_cg.cuh)
static constexpr int kXMarchVariant = kNumVariants + 1;  // streamed, vectors x2-fastest (xmarch.cuh)
static constexpr int kAllVariants = kNumVariants + 2;

// Ring-march instances per n1: (x2 tile capacity, register cap per thread)
// of its two variants. A CTA's threads x registers must fit the SM's 65,536,
// with registers counted in units of 16 per thread (136 measured as too many
// for 480 threads); 128 registers spill a few bytes.
template <int N1> struct RingTraits;
// Variant A unrolls the march over the ring; variant B is the same tile
// without the unrolling (DYN: smaller code, window moves).
template <> struct RingTraits<9> { static constexpr int T2A = 7, MA = 128, T2B = 7, MB = 128; };
template <> struct RingTraits<21> { static constexpr int T2A = 7, MA = 128, T2B = 7, MB = 128; };
template <> struct RingTraits<33> { static constexpr int T2A = 7, MA = 96, T2B = 7, MB = 96; };
static_assert(ring_threads(9, RingTraits<9>::T2B) * RingTraits<9>::MB <= 65536, "ring CTA exceeds the register file");
static_assert(ring_threads(21, RingTraits<21>::T2B) * RingTraits<21>::MB <= 65536, "ring CTA exceeds the register file");
static_assert(ring_threads(33, RingTraits<33>::T2A) * RingTraits<33>::MA <= 65536, "ring CTA exceeds the register file");
static_assert(ring_threads(33, RingTraits<33>::T2B) * RingTraits<33>::MB <= 65536, "ring CTA exceeds the register file");

// The largest CTA the device will launch for a ring-march instance (its
// register use included).
template <int N1>
static int ring_max_threads(int which) {
    using R = RingTraits<N1>;
    cudaFuncAttributes fa{};
    cudaError_t e = which == 0 ? cudaFuncGetAttributes(&fa, ring_march_kernel<N1, R::T2A, R::MA>)
                               : cudaFuncGetAttributes(&fa, ring_march_kernel<N1, R::T2B, R::MB, true>);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return fa.maxThreadsPerBlock;
}

static int ring_launchable_threads(int n1, int which) {
    switch (n1) {
    case 9: return ring_max_threads<9>(which);
    case 21: return ring_max_threads<21>(which);
    case 33: return ring_max_threads<33>(which);
    default: return 0;
    }
}

static int ring_t2_for(int n1, int which) {
    switch (n1) {
    case 9: return which == 0 ? RingTraits<9>::T2A : RingTraits<9>::T2B;
    case 21: return which == 0 ? RingTraits<21>::T2A : RingTraits<21>::T2B;
    case 33: return which == 0 ? RingTraits<33>::T2A : RingTraits<33>::T2B;
    default: return 0;
    }
}

// Launch configuration of ring_march_kernel: 7-row tiles at both x2 ends,
// the rows between split into tiles of at most t2 rows.
static bool make_ring_cfg(const GridConst &gc, const double h[3], int which, MarchCfg &out, std::string &why) {
    const int t2 = ring_t2_for(gc.n1, which);
    if (t2 <= 0) {
        why = "ring march: n1 = " + std::to_string(gc.n1) + " has no specialised instance";
        return false;
    }
    if (gc.n2 < 2 * kRingEdge) {
        why = "ring march: n2 below 14";
        return false;
    }
    if (ring_threads(gc.n1, t2) > ring_launchable_threads(gc.n1, which)) {
        why = "ring march: the CTA does not fit the device's register file";
        return false;
    }
    const int m = gc.n2 - 2 * kRingEdge;
    const int nmid = m > 0 ? (m + t2 - 1) / t2 : 0;
    out = MarchCfg{};
    out.ring_t2 = t2;
    out.ring_var = which;
    out.rg.n2 = gc.n2;
    out.rg.n3 = gc.n3;
    out.rg.PS = gc.PS;
    out.rg.colstride = gc.colstride;
    out.rg.ntiles = nmid + 2;
    out.rg.nmid = std::max(nmid, 1);
    out.rg.drop_plane = -1;
    out.rg.poll_limit = 0;
    {
        const double lam = gc.lam, mu = gc.mu, lpm = gc.lam + gc.mu;
        const double h2 = h[1], h3 = h[2], h2i = 1.0 / h2, h3i = 1.0 / h3;
        RingScal &k = out.rg.k;
        k.lam = (float)lam;
        k.mu = (float)mu;
        k.mu2 = (float)(2 * mu);
        k.lpm = (float)lpm;
        k.lpm_h2 = (float)(lpm * h2i);
        k.lpm_h3 = (float)(lpm * h3i);
        k.lam_h2 = (float)(lam * h2i);
        k.lam_h3 = (float)(lam * h3i);
        k.mu_h2 = (float)(mu * h2i);
        k.mu_h3 = (float)(mu * h3i);
        k.mu_h2s = (float)(mu * h2i * h2i);
        k.mu2_h2s = (float)(2 * mu * h2i * h2i);
        k.lam_h2s = (float)(lam * h2i * h2i);
        k.mu_h3s = (float)(mu * h3i * h3i);
        k.mu2_h3s = (float)(2 * mu * h3i * h3i);
        k.lpm_h2h3 = (float)(lpm * h2i * h3i);
        k.h3i = (float)h3i;
        k.h2 = (float)h2;
        k.h2s = (float)(h2 * h2);
        k.h3 = (float)h3;
        k.h3s = (float)(h3 * h3);
        k.sat = (float)gc.sat_c;
    }
    out.g.n1 = gc.n1;
    out.g.n2 = gc.n2;
    out.g.n3 = gc.n3;
    out.g.PS = gc.PS;
    out.g.colstride = gc.colstride;
    out.g.ntiles = out.rg.ntiles;
    out.g.t2max = t2;
    out.g.nblk = 1;
    out.g.nseg = 1;
    out.g.segblk = 1;
    out.g.target = 0;
    out.g.edge = kRingEdge;
    out.threads = ring_threads(gc.n1, t2);
    out.smem = ring_smem(gc.n1, t2);
    out.smem_af = 0;  // the direction update is not fused into this kernel
    return true;
}

static bool n1_specialized(int n1) { return n1 == 9 || n1 == 21 || n1 == 33; }

// `maxt` limits the threads of the tile; `kmaxt` is the launch bound of the
// kernel instance that will run it (it fixes the shared-memory geometry of
// the n1-specialized instances).
template <typename T>
static bool make_march_cfg(int n1, int n2, int n3, int PS, long long colstride, int maxt, int tile_rows,
                           const GridConst &gc, MarchCfg &out, std::string &why, int lanes = 1, int kmaxt = 0,
                           bool edge_mode = false) {
    if (kmaxt == 0) kmaxt = maxt;
    const int per_row = 2 * n1;
    int t2 = tile_rows > 0 ? std::min(tile_rows, maxt / per_row) : maxt / per_row;
    t2 = std::min(t2, n2);
    if (t2 * per_row > maxt) t2 = maxt / per_row;
    int ntiles = (n2 + t2 - 1) / t2;
    if (ntiles < 1) ntiles = 1;
    // Balanced tiles, every tile at least 7 rows: the wide operator's closure
    // rows reach 10 rows in from the boundary, and a tile reads 4 halo rows.
    while (ntiles > 1 && n2 / ntiles < 7) --ntiles;
    int t2max = (n2 + ntiles - 1) / ntiles;
    int edge = 0;
    // Edge partition: forced (a launch variant that keeps every x2 closure row
    // in 7-row edge tiles, so no CTA mixes closure and interior rows), or
    // needed when balanced tiles of >= 7 rows do not fit the thread limit.
    if ((edge_mode || t2max * per_row > maxt) && t2 >= 7 && n2 >= 14) {
        // Tiles of at most t2 rows: 7-row tiles at both ends carry the closure
        // rows, the tiles between (any height) split the interior.
        edge = 7;
        const int m = n2 - 2 * edge;
        const int nm = m > 0 ? (m + t2 - 1) / t2 : 0;
        ntiles = nm + 2;
        t2max = std::max(edge, nm > 0 ? (m + nm - 1) / nm : 0);
    }
    if (t2max * per_row > maxt || (edge == 0 && n2 / ntiles < std::min(7, n2))) {
        why = "grid too large in x1 for one CTA (n1=" + std::to_string(n1) + ")";
        return false;
    }
    constexpr int AE = 16 / (int)sizeof(T);
    int CH = (t2max + 2 * EQD_HALO) * n1 + 2 * AE;
    CH = (CH + AE - 1) / AE * AE;
    int NP = 2 * n1 * t2max;
    if (n1_specialized(n1)) {
        if (t2max > march_t2cap(n1, kmaxt)) {
            why = "tile exceeds the specialized kernel's capacity";
            return false;
        }
        CH = march_chcap(n1, kmaxt, (int)sizeof(T));
        NP = 2 * n1 * march_t2cap(n1, kmaxt);
    }
    out.g.n1 = n1;
    out.g.n2 = n2;
    out.g.n3 = n3;
    out.g.PS = PS;
    out.g.colstride = colstride;
    out.g.ntiles = ntiles;
    out.g.t2max = t2max;
    out.g.edge = edge;
    out.g.CH = CH;
    out.g.i2f0 = gc.i2f0;
    out.g.n2f = gc.n2f;
    out.g.i3f0 = gc.i3f0;
    out.g.n3f = gc.n3f;
    out.g.nf = gc.nf;
    // FP64-input instances sum dot products per x3 step block (and can split
    // a column along x3); FP32 ones per tile over the whole column.
    out.g.nblk = sizeof(T) == 8 ? (n3 + EQD_PBLK - 1) / EQD_PBLK : 1;
    out.g.nseg = 1;
    out.g.segblk = out.g.nblk;
    out.g.target = 0;
    int threads = per_row * t2max;
    threads = (threads + 31) / 32 * 32;
    out.threads = threads;
    // barriers + flags, reduction scratch, and per column: plane ring, F1/H21
    // exchange [2][points] x 2; FP64: per-(step block, warp) dot-product sums
    out.smem = 64 + 32 * 8 + (size_t)lanes * ((size_t)EQD_NSLOT * 6 * CH + 4 * (size_t)NP) * sizeof(T);
    if (sizeof(T) == 8) out.smem += 16 + (size_t)lanes * out.g.nblk * (threads / 32) * 2 * sizeof(double);
    // MODE_AF adds the ring of r planes (aligned to 128 bytes after the rest).
    out.smem_af = out.smem + 144 + (size_t)lanes * EQD_NSLOT * 6 * CH * sizeof(T);
    return true;
}

// Dot-product partials per column of a launch configuration: one per
// (x2 tile, x3 step block) for FP64-input configurations, one per x2 tile
// for FP32 ones (nblk = 1).
static int nparts(const MarchCfg &m) { return m.g.ntiles * m.g.nblk; }

// x3 segmentation of an FP64-input launch: a batch too small to give every
// SM two CTAs is split along x3 into segments of whole step blocks (a
// segment marches 9 to 14 planes before its first block to fill its windows
// and 3 planes past its last). Partials are per step block, so the results
// do not depend on the split.
static MarchCfg segmented(const MarchCfg &m, long long groups, int num_sms) {
    MarchCfg r = m;
    const long long ctas = groups * m.g.ntiles;
    const long long target = 2LL * num_sms;
    if (ctas >= target || m.g.nblk <= 1) return r;
    const int want = (int)std::min<long long>((target + ctas - 1) / ctas, m.g.nblk);
    r.g.segblk = (m.g.nblk + want - 1) / want;
    r.g.nseg = (m.g.nblk + r.g.segblk - 1) / r.g.segblk;
    return r;
}

// Columns that a launch is split for: with flags (reliable updates, columns
// that enter) as many as are flagged in most iterations, a column in 64 (five
// times in about 320) and at least four; where more are flagged the kernel
// joins segments again, and where none is, more CTAs would only have to leave.
static int flagged_cols(const ColumnSet &cs, int ncols) {
    return cs.flag ? std::min(ncols, std::max(4, ncols / 64)) : ncols;
}

template <typename T>
static void fill_op(OpConst<T> &C, const GridConst &gc, const double h[3]) {
    for (int a = 0; a < 3; ++a) fill_axis<T>(C.ax[a], a == 0 ? gc.n1 : (a == 1 ? gc.n2 : gc.n3), h[a]);
    C.lam = (T)gc.lam;
    C.mu = (T)gc.mu;
    C.lpm = (T)(gc.lam + gc.mu);
    C.sat_c = (T)gc.sat_c;
    C.hvol = gc.hvol;
}

// Page-locked host array: device-to-host copies into it stay asynchronous.
template <typename E>
struct PinnedArr {
    E *p = nullptr;
    int n = 0;
    PinnedArr() = default;
    PinnedArr(const PinnedArr &) = delete;
    PinnedArr &operator=(const PinnedArr &) = delete;
    ~PinnedArr() {
        if (p) cudaFreeHost(p);
    }
    cudaError_t assign(int count, E v) {
        if (count > n) {
            if (p) cudaFreeHost(p);
            p = nullptr;
            n = 0;
            cudaError_t e = cudaHostAlloc((void **)&p, sizeof(E) * std::max(count, 1), cudaHostAllocDefault);
            if (e != cudaSuccess) return e;
            n = count;
        }
        for (int i = 0; i < count; ++i) p[i] = v;
        return cudaSuccess;
    }
    E *data() { return p; }
    E &operator[](int i) { return p[i]; }
    const E &operator[](int i) const { return p[i]; }
};

// Workspace of one batched solve (grown on demand, reused across calls).
struct Workspace {
    int cap = 0;            // columns
    int precision = -1;
    DevBuf x64, v0, v1, v2, v3;  // x64 + (r, p, q, d) in the working precision
    DevBuf v4;                   // fused direction update: the other p buffer (p alternates v1, v4)
    DevBuf apply_part, res_part, rr_part;
    DevBuf gamma, beta, rr_ref, tol, bnorm, pp, iters, status, flag;
    DevBuf slip_node, slip_comp, slip_dense;
    DevBuf kout;
    DevBuf newmask, slot_list, dst_list;  // slot engine: entering columns, extraction lists
    DevBuf hbuf;                          // explicit-RHS staging (reference layout)
    PinnedArr<double> kstage;             // finished K columns on their way to a host K
    cudaGraphExec_t graph = nullptr;
    int graph_iters = 0;
    bool graph_split = false;  // the captured iterations run as two halves
    CUtensorMap pmap;          // x1 march: the planes of p
    std::vector<uint64_t> graph_key;  // what the captured graph baked in (see SlotRun::setup)
    ~Workspace() {
        if (graph) cudaGraphExecDestroy(graph);
    }
};

// The resident CG of one precision: its plan, the device tables, and the
// kernel instance that runs it.
struct ResEngine {
    bool tried = false, ok = false;
    ResDims d{};
    int t2 = 0, t3 = 0;  // tile capacity of the kernel instance
    int teams = 0;       // > 0: teams that meet through global memory (else one cluster a column)
    bool few = false;    // the teams are for a few explicit right-hand sides only
    DevBuf ranks, chunks, lines, gofs, push, pull, tab, off, team_p, team_red, team_count;
    ResTables tb{};
};

// The streamed FP32 iteration on x2-fastest vectors: geometry and tables.
struct XEngine {
    bool tried = false, ok = false;
    XGeom g{};
    XCoef C{};
    XLayout lay{};
    int smem = 0;
    int nchunks = 1;  // of a column in cg_step_bulk_kernel
    DevBuf b2, b3, rows, tab, off;
};

struct eqd_grid {
    eqd_grid_desc desc;
    GridConst gc;
    double h[3];
    OpConst<float> c32;
    OpConst<double> c64;
    MarchCfg m32, m64;
    int m64_maxt = 384;   // launch bound of the FP64 instance the grid runs
    bool served = false;  // attached to an eqd_server (its worker owns the grid)
    int num_sms = 148;
    DevBuf dinv64, dinv32;   // Jacobi weights (one column, device layout)
    bool jacobi_ready = false;
    // FP32 A-apply launch variants (see make_variants) and the chosen one.
    MarchCfg v32[kNumVariants];
    int v32_maxt[kNumVariants] = {};
    int v32_lanes[kNumVariants] = {};
    int sel32 = 0;
    bool tuned = false;
    int pin = -1;          // variant the caller (or eqd_autotune) chose, kResidentVariant included; -1: none,
                           // and solves run resident where the grid has a plan
    int pin64 = -1;        // the same for FP64 solves, the caller's only: the tuner times mixed precision
    ResEngine res32, res64;
    XEngine xm;
    int chunk_tuned = 0;   // eqd_tune_chunk's choice of columns per batch (0: as many as the budget allows)
    double tune_ms[kAllVariants] = {};
    int nchunks = 1;
    cudaStream_t stream = nullptr;
    cudaStream_t stream2 = nullptr;          // second half of a split batch (graph capture only)
    cudaStream_t stream_hi = nullptr, stream2_hi = nullptr;  // high priority: vector kernels of the halves
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t evA = nullptr, evB = nullptr, evFork = nullptr, evJoin = nullptr, evArest = nullptr,
                evBrest = nullptr;
    DevBuf err;           // device error word
    Workspace ws;
    std::mutex mtx;
    std::vector<double> x2f, x3f;
    int tile_rows = 0;
    bool test_fail_launch = false; // eqd_test_inject_failure: the next CG launch that is recorded fails on the host
    bool test_fail_plan = false;   // and the next allocation for the tables of a plan
    int test_drop_plane = -1;      // eqd_test_inject_wait_timeout: the next ring launch never copies this plane
    unsigned test_poll_limit = 0;
};

struct eqd_kmat {
    int device;
    int n;
    int ks_slots[3] = {296, 296, 296};  // resident CTAs of the blocked K S (16, 32, 64 vectors per CTA)
    DevBuf K, s, y, part;
    cudaStream_t stream = nullptr;
};

// ---------------------------------------------------------------------------
// Kernel launch helpers
// ---------------------------------------------------------------------------
// Kernel instances compiled for a fixed n1 (the BP8 grids' 9, 21, 33 points
// across a side); any other n1 runs the runtime-n1 instance.
#define EQD_FOR_N1(X) X(9) X(21) X(33)

template <typename T, typename TO, int MODE, int MAXT, int L = 1>
static void launch_n1(int n1, dim3 grid, const MarchCfg &m, cudaStream_t st, const OpConst<T> &C, const T *in,
                      TO *out, ColumnSet cs, double *partials, unsigned *err) {
    switch (n1) {
#define EQD_CASE(N)                                                                                       \
    case N:                                                                                               \
        plane_march_kernel<T, TO, MODE, MAXT, N, L><<<grid, m.threads, m.smem, st>>>(C, m.g, in, out, cs, \
                                                                                     partials, err);      \
        return;
        EQD_FOR_N1(EQD_CASE)
#undef EQD_CASE
    default:
        plane_march_kernel<T, TO, MODE, MAXT, 0, L><<<grid, m.threads, m.smem, st>>>(C, m.g, in, out, cs,
                                                                                     partials, err);
    }
}

template <int N1>
static void launch_ring_n1(int which, dim3 grid, const MarchCfg &m, const RingGeom &rg, cudaStream_t st,
                           const OpConst<float> &C, const float *in, float *out, const int8_t *status,
                           double *partials, unsigned *err) {
    using R = RingTraits<N1>;
    if (which == 0)
        ring_march_kernel<N1, R::T2A, R::MA><<<grid, m.threads, m.smem, st>>>(C, rg, in, out, status, partials, err);
    else
        ring_march_kernel<N1, R::T2B, R::MB, true><<<grid, m.threads, m.smem, st>>>(C, rg, in, out, status, partials,
                                                                                     err);
}

// The FP32 CG apply through ring_march_kernel (one CTA per column and x2
// tile). A pending test injection (eqd_test_inject_wait_timeout) applies to
// this launch only.
static cudaError_t launch_ring(eqd_grid *G, const MarchCfg &m, const float *in, float *out, const ColumnSet &cs,
                               double *partials, int ncols, cudaStream_t st) {
    RingGeom rg = m.rg;
    if (G->test_drop_plane >= 0) {
        rg.drop_plane = G->test_drop_plane;
        rg.poll_limit = G->test_poll_limit;
        G->test_drop_plane = -1;
    }
    const dim3 grid((unsigned)((long long)ncols * rg.ntiles));
    unsigned *err = G->err.as<unsigned>();
    switch (G->gc.n1) {
    case 9: launch_ring_n1<9>(m.ring_var, grid, m, rg, st, G->c32, in, out, cs.status, partials, err); break;
    case 21: launch_ring_n1<21>(m.ring_var, grid, m, rg, st, G->c32, in, out, cs.status, partials, err); break;
    case 33: launch_ring_n1<33>(m.ring_var, grid, m, rg, st, G->c32, in, out, cs.status, partials, err); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename T, typename TO, int MODE>
static cudaError_t launch_march(eqd_grid *G, const T *in, TO *out, ColumnSet cs, double *partials, int ncols,
                                int variant = -1, cudaStream_t stream = nullptr) {
    cs.ncols = ncols;
    cudaStream_t st = stream ? stream : G->stream;
    const int n1 = G->gc.n1;
    if constexpr (sizeof(T) == 4 && (MODE == MODE_A || MODE == MODE_AF)) {
        const int v = variant >= 0 ? variant : G->sel32;
        if (G->v32[v].ring_t2 > 0) {
            if (MODE == MODE_AF) return cudaErrorInvalidValue;  // not fused in this kernel (smem_af = 0)
            return launch_ring(G, G->v32[v], reinterpret_cast<const float *>(in), reinterpret_cast<float *>(out), cs,
                               partials, ncols, st);
        }
        const int lanes = G->v32_lanes[v];
        const long long groups = (ncols + lanes - 1) / lanes;
        MarchCfg m = segmented(G->v32[v], groups, G->num_sms);
        if (MODE == MODE_AF) m.smem = m.smem_af;
        dim3 grid((unsigned)(groups * m.g.ntiles * m.g.nseg));
        const float *fin = reinterpret_cast<const float *>(in);
        float *fout = reinterpret_cast<float *>(out);
        if (lanes == 2)
            launch_n1<float, float, MODE, kMaxT32c, 2>(n1, grid, m, st, G->c32, fin, fout, cs, partials,
                                                        G->err.as<unsigned>());
        else if (G->v32_maxt[v] == kMaxT32)
            launch_n1<float, float, MODE, kMaxT32>(n1, grid, m, st, G->c32, fin, fout, cs, partials,
                                                   G->err.as<unsigned>());
        else
            launch_n1<float, float, MODE, kMaxT32b>(n1, grid, m, st, G->c32, fin, fout, cs, partials,
                                                    G->err.as<unsigned>());
        return cudaGetLastError();
    }
    constexpr int MAXT = sizeof(T) == 4 ? kMaxT32 : kMaxT64;
    MarchCfg m = segmented(sizeof(T) == 4 ? G->m32 : G->m64, MODE == MODE_RHS ? flagged_cols(cs, ncols) : ncols, G->num_sms);
    if (MODE == MODE_RHS && sizeof(T) == 8 && cs.flag) m.g.target = 2 * G->num_sms;
    if (MODE == MODE_AF) m.smem = m.smem_af;
    const OpConst<T> &C = *reinterpret_cast<const OpConst<T> *>(sizeof(T) == 4 ? (const void *)&G->c32
                                                                               : (const void *)&G->c64);
    dim3 grid((unsigned)(ncols * m.g.ntiles * m.g.nseg));
    const bool wide64 = sizeof(T) == 8 && G->m64_maxt == kMaxT64b;
    if (MODE == MODE_AP) {  // generic-input hook: runtime-n1 instance only
        if (wide64)
            plane_march_kernel<T, TO, MODE, kMaxT64b, 0, 1><<<grid, m.threads, m.smem, st>>>(
                C, m.g, in, out, cs, partials, G->err.as<unsigned>());
        else
            plane_march_kernel<T, TO, MODE, MAXT, 0, 1><<<grid, m.threads, m.smem, st>>>(
                C, m.g, in, out, cs, partials, G->err.as<unsigned>());
    } else if (wide64) {
        launch_n1<T, TO, MODE, kMaxT64b>(n1, grid, m, st, C, in, out, cs, partials, G->err.as<unsigned>());
    } else {
        launch_n1<T, TO, MODE, MAXT>(n1, grid, m, st, C, in, out, cs, partials, G->err.as<unsigned>());
    }
    return cudaGetLastError();
}

// Dynamic shared memory above 48 KB must be opted into per kernel.
static cudaError_t configure_kernels(int smem_max) {
#define EQD_KS(N)                                                                \
    (const void *)plane_march_kernel<float, float, MODE_A, kMaxT32, N, 1>,       \
        (const void *)plane_march_kernel<float, float, MODE_A, kMaxT32b, N, 1>,    \
        (const void *)plane_march_kernel<float, float, MODE_A, kMaxT32c, N, 2>,    \
        (const void *)plane_march_kernel<float, float, MODE_RHS, kMaxT32, N, 1>,   \
        (const void *)plane_march_kernel<double, double, MODE_A, kMaxT64, N, 1>,   \
        (const void *)plane_march_kernel<double, double, MODE_RHS, kMaxT64, N, 1>, \
        (const void *)plane_march_kernel<double, float, MODE_RHS, kMaxT64, N, 1>,   \
        (const void *)plane_march_kernel<double, double, MODE_A, kMaxT64b, N, 1>,  \
        (const void *)plane_march_kernel<double, double, MODE_RHS, kMaxT64b, N, 1>, \
        (const void *)plane_march_kernel<double, float, MODE_RHS, kMaxT64b, N, 1>,       \
        (const void *)plane_march_kernel<float, float, MODE_AF, kMaxT32, N, 1>,          \
        (const void *)plane_march_kernel<float, float, MODE_AF, kMaxT32b, N, 1>,         \
        (const void *)plane_march_kernel<float, float, MODE_AF, kMaxT32c, N, 2>,         \
        (const void *)plane_march_kernel<double, double, MODE_AF, kMaxT64, N, 1>,        \
        (const void *)plane_march_kernel<double, double, MODE_AF, kMaxT64b, N, 1>,
#define EQD_RING_KS(N)                                                                                     \
    (const void *)ring_march_kernel<N, RingTraits<N>::T2A, RingTraits<N>::MA>,                             \
        (const void *)ring_march_kernel<N, RingTraits<N>::T2B, RingTraits<N>::MB, true>,
    const void *ks[] = {
        EQD_FOR_N1(EQD_KS) EQD_KS(0)
        (const void *)plane_march_kernel<float, float, MODE_AP, kMaxT32, 0, 1>,
        (const void *)plane_march_kernel<double, double, MODE_AP, kMaxT64, 0, 1>,
        (const void *)plane_march_kernel<double, double, MODE_AP, kMaxT64b, 0, 1>,
        EQD_FOR_N1(EQD_RING_KS)
    };
#undef EQD_RING_KS
#undef EQD_KS
    for (const void *k : ks) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Resident CG (resident_cg.cuh): plan, tables and launch
// ---------------------------------------------------------------------------
// Kernel instances: n1, the largest tile of own lines, and the parts that a
// line is cut into. The x1 lines of the BP8 grids at 100, 80, 50 and 40 m (9 to
// 21 points) and of the cubes up to 25. The last number: 0, one cluster to a
// column; 1, a team that meets through global memory, for a few explicit
// right-hand sides, up to four a team (25^3: one 5.3 ms against 22, 12 32
// against 45); 2, for columns too where team_fills. Where it does not, the
// streamed iteration is the better one for many (25^3, 300 columns: 243 ms
// against 579), and the choice for columns does not depend on
// their number, so that a column's bits do not either. FP32 teams, tried at
// 17 and 21 points, halve a single column's time (h = 40 m 6.8 ms against
// 15.3) but lose from 16 on (h = 20 m, 64 columns: 548 ms against 220).
#define EQD_RES_32(X) \
    X(9, 8, 8, 2, 0) X(9, 8, 16, 2, 0) X(11, 8, 8, 2, 0) X(11, 8, 16, 2, 0) X(13, 8, 8, 2, 0) X(15, 8, 8, 2, 0) \
    X(17, 8, 8, 2, 0) X(21, 8, 8, 2, 0) X(25, 8, 8, 2, 0)
#define EQD_RES_64(X) \
    X(9, 8, 8, 2, 0) X(11, 8, 8, 2, 0) X(13, 8, 8, 2, 0) X(15, 8, 4, 3, 0) X(17, 8, 4, 4, 0) X(19, 8, 4, 4, 0) \
    X(17, 8, 4, 4, 2) X(19, 8, 4, 4, 1) X(21, 7, 4, 4, 1) X(23, 4, 4, 4, 1) X(25, 4, 4, 4, 1) X(27, 4, 4, 5, 1) \
    X(29, 4, 3, 5, 1)

template <int N1, int T2, int T3, int NP, int GRID>
struct ResInstance {
    static constexpr int n1 = N1, t2 = T2, t3 = T3, np = NP;
    static constexpr bool grid = GRID > 0, few = GRID == 1;
    template <typename T>
    static constexpr auto kernel() {
        return resident_cg_kernel<T, N1, T2, T3, NP, grid>;
    }
};

// f(ResInstance) for the instances of precision T in turn, until one returns true.
template <typename T, typename F>
static bool res_instances(F &&f) {
#define EQD_CASE(N, A, B, P, R) f(ResInstance<N, A, B, P, R>()) ||
    if constexpr (sizeof(T) == 4) return EQD_RES_32(EQD_CASE) false;
    else return EQD_RES_64(EQD_CASE) false;
#undef EQD_CASE
}

// Warps of a CTA: one per part of a line and chunk of own lines; a team that
// meets through global memory is small per CTA and has halo rows done by more.
static int res_warps(const ResDims &d, int np, bool grid, int most) {
    const int own = np * d.nch0max;
    return grid ? std::max(own, std::min(most, np * d.nhalomax)) : own;
}

static void res_launch_config(const ResDims &d, int warps, int teams, bool grid, cudaStream_t s,
                              cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at) {
    cfg = cudaLaunchConfig_t{};
    at = cudaLaunchAttribute{};
    if (grid) {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    } else {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)d.M;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    }
    cfg.gridDim = dim3((unsigned)teams * (unsigned)d.M);
    cfg.blockDim = dim3((unsigned)(32 * warps));
    cfg.dynamicSmemBytes = (size_t)d.smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}

// A table of a plan, on the device. (A plan that an error cut short is made anew
// by the next call: a grid keeps to one kernel, and so a column to its bits.)
static cudaError_t put_table(eqd_grid *G, DevBuf &b, const void *src, size_t bytes) {
    if (G->test_fail_plan) {
        G->test_fail_plan = false;
        return cudaErrorMemoryAllocation;
    }
    const cudaError_t e = b.ensure(std::max<size_t>(bytes, 16));
    return e == cudaSuccess && bytes ? cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, G->stream) : e;
}

// Whether teams of M CTAs keep up with the streamed iteration for hundreds of
// columns: 25 own lines for every SM of the device, and four teams at least
// (larger ones wait longer for one another). FP64, 17 points, 300 columns,
// streamed against teams: 33 x 33 nodes (26 lines, 4 teams) 220 ms against 208;
// 25 x 33 (24, 5) 197, 190; 33 x 25 (24, 5) 161, 167; 41 x 33 (24.5, 3) 290, 339;
// 29 x 29 (20, 4) 166, 211; 65 x 33 (26, 2) 452, 558; 49 x 17 (19, 4) 148, 183.
// At 33 x 33 six columns take 3.2 ms against 21, 40 28 against 49, and 1,000 687
// against 611: the price of one path for every number of columns.
static bool team_fills(const GridConst &gc, int M, int num_sms) {
    const int teams = num_sms / M;
    return teams >= 4 && (long long)(gc.n2 - 2) * (gc.n3 - 2) * teams >= 25LL * num_sms;
}

// The team and the instance with the least work per column-iteration over the
// team (whole K at h = 50 m: 8 CTAs of 8 x 16 lines 205 ms, 16 of 8 x 8 227 ms;
// h = 100 m: 2 of 8 x 16 9.2 ms, 4 of 8 x 8 9.9 ms, 9 of them 15.1 ms).
template <typename T>
static int ensure_resident(eqd_grid *G, ResEngine &E) {
    if (E.tried) return EQD_OK;
    const GridConst &gc = G->gc;
    ResPlan best;
    double best_cost = 1e300;
    res_instances<T>([&](auto I) {
        if (I.n1 != gc.n1 || (I.grid && best_cost < 1e300)) return false;  // a cluster is listed, and taken, first
        const void *k = (const void *)I.template kernel<T>();
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, k) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmemMax) != cudaSuccess ||
            (!I.grid && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
            cudaGetLastError();
            return false;
        }
        const auto strides = res_strides<sizeof(T), I.n1, I.t2, I.t3>();
        auto consider = [&](int m2, int m3) {
            ResPlan P;
            if (!make_res_plan(gc.n1, gc.n2, gc.n3, gc.PS, m2, m3, strides, P, I.grid)) return;
            const int warps = res_warps(P.d, I.np, I.grid, fa.maxThreadsPerBlock / 32);
            if (32 * warps > fa.maxThreadsPerBlock || P.cost >= best_cost) return;
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at;
            res_launch_config(P.d, warps, 1, I.grid, nullptr, cfg, at);
            int fit = 0;
            if (I.grid) {
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, 32 * warps, P.d.smem) != cudaSuccess) fit = 0;
                fit = fit * G->num_sms / P.d.M;
            } else if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess) {
                fit = 0;
            }
            cudaGetLastError();  // (the device cannot place this cluster)
            if (fit < 1) return;
            best_cost = P.cost;
            best = P;
            E.t2 = I.t2;
            E.t3 = I.t3;
            E.teams = I.grid ? fit : 0;
            E.few = I.few || (I.grid && !team_fills(gc, P.d.M, G->num_sms));
        };
        if (I.grid) {  // the fewest tiles that fit
            int m[2] = {1, 1};
            const int n[2] = {gc.n2, gc.n3}, most[2] = {I.t2, I.t3};
            for (int a = 0; a < 2; ++a)
                for (; m[a] <= kResMaxGridTeam; ++m[a]) {
                    std::vector<int> b;
                    if (!res_split(n[a], m[a], b)) continue;
                    int w = 0;
                    for (int q = 0; q < m[a]; ++q) w = std::max(w, b[q + 1] - b[q]);
                    if (w <= most[a]) break;
                }
            if (m[0] * m[1] <= kResMaxGridTeam) consider(m[0], m[1]);
        } else {
            for (int m2 = 1; m2 <= kResMaxTeam; ++m2)
                for (int m3 = 1; m2 * m3 <= kResMaxTeam; ++m3) consider(m2, m3);
        }
        return false;
    });
    std::vector<T> tab;
    std::vector<int> off;
    if (best_cost == 1e300 || !fill_res_tables<T>(gc.n2, gc.n3, G->h[1], G->h[2], gc.mu, tab, off)) {
        E.tried = true;
        return EQD_OK;
    }
    E.d = best.d;
    auto put = [&](DevBuf &b, const void *src, size_t bytes) { return put_table(G, b, src, bytes); };
    CUDA_OR_RETURN(put(E.ranks, best.ranks.data(), best.ranks.size() * sizeof(ResRank)));
    CUDA_OR_RETURN(put(E.chunks, best.chunks.data(), best.chunks.size() * sizeof(int)));
    CUDA_OR_RETURN(put(E.lines, best.lines.data(), best.lines.size() * sizeof(ResLine)));
    CUDA_OR_RETURN(put(E.gofs, best.gofs.data(), best.gofs.size() * sizeof(int)));
    CUDA_OR_RETURN(put(E.push, best.push.data(), best.push.size() * sizeof(int)));
    CUDA_OR_RETURN(put(E.pull, best.pull.data(), best.pull.size() * sizeof(ResPull)));
    CUDA_OR_RETURN(put(E.tab, tab.data(), tab.size() * sizeof(T)));
    CUDA_OR_RETURN(put(E.off, off.data(), off.size() * sizeof(int)));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    E.tb = ResTables{E.ranks.as<ResRank>(), E.chunks.as<int>(), E.lines.as<ResLine>(), E.gofs.as<int>(),
                     E.push.as<int>(), E.pull.as<ResPull>(), E.tab.p, E.off.as<int>()};
    if (E.teams) {
        const size_t ctas = (size_t)E.teams * E.d.M;
        size_t cs = 0;
        res_instances<T>([&](auto I) {
            if (I.grid && I.n1 == gc.n1 && I.t2 == E.t2 && I.t3 == E.t3)
                cs = ResGeo<sizeof(T), I.n1, I.t2, I.t3>::CS;
            return cs > 0;
        });
        CUDA_OR_RETURN(E.team_p.ensure(sizeof(T) * 3 * cs * ctas));
        CUDA_OR_RETURN(E.team_red.ensure(sizeof(double) * 8 * ctas));
        CUDA_OR_RETURN(E.team_count.ensure(sizeof(unsigned) * 32 * E.teams));
        // (never written, or only read by a CTA that owns none: the far rows of a tile)
        CUDA_OR_RETURN(cudaMemsetAsync(E.team_p.p, 0, sizeof(T) * 3 * cs * ctas, G->stream));
        CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    }
    E.tried = E.ok = true;
    return EQD_OK;
}

// Up to kmax iterations of every active column (x: the FP32 correction, or
// the FP64 solution).
template <typename T>
static cudaError_t launch_resident(eqd_grid *G, const ResEngine &E, T *x, T *r, T *p, const ColState &st,
                                   const SolveParams &sp, int mixed, int kmax, int ncols, cudaStream_t s) {
    cudaError_t e = cudaErrorInvalidValue;
    res_instances<T>([&](auto I) {
        if (I.n1 != G->gc.n1 || I.t2 != E.t2 || I.t3 != E.t3 || I.grid != (E.teams > 0)) return false;
        const auto k = I.template kernel<T>();
        cudaFuncAttributes fa{};
        e = cudaFuncGetAttributes(&fa, (const void *)k);
        if (e != cudaSuccess) return true;
        const int teams = I.grid ? std::min(ncols, E.teams) : ncols;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        res_launch_config(E.d, res_warps(E.d, I.np, I.grid, fa.maxThreadsPerBlock / 32), teams, I.grid, s, cfg, at);
        const ResCoef<T> C = res_coef<T>(G->h[0], G->gc.lam, G->gc.mu, G->gc.sat_c);
        const ResX1<T, I.n1> X = res_x1<T, I.n1>(G->h[0], G->gc.mu, G->gc.hvol);
        ResTeam<T> team{};
        if constexpr (I.grid) {
            team = ResTeam<T>{E.team_p.template as<T>(), E.team_red.template as<double>(),
                              E.team_count.template as<unsigned>(), teams, G->err.as<unsigned>()};
            e = cudaMemsetAsync(team.count, 0, sizeof(unsigned) * 32 * teams, s);
            if (e != cudaSuccess) return true;
        }
        e = cudaLaunchKernelEx(&cfg, k, C, X, E.d, E.tb, x, r, p, st, sp, mixed, kmax, ncols, team);
        return true;
    });
    return e;
}

// ---------------------------------------------------------------------------
// x1 march (xmarch.cuh): tiles, tables, tensor map and launch
// ---------------------------------------------------------------------------
static int ensure_xmarch(eqd_grid *G) {
    XEngine &E = G->xm;
    if (E.tried) return EQD_OK;
    const GridConst &gc = G->gc;
    std::vector<int> b2, b3, off;
    std::vector<float> tab, rows((size_t)gc.n1 * 16, 0.f);
    // Tiles start every fourth line along x2 (a tiled copy starts on 16 bytes).
    if (!x_offsets_fit(gc.n1, gc.n2, gc.n3) || !x_tiles(gc.n2, 1, kXT2, 4, b2) || !x_tiles(gc.n3, 1, kXT3, 1, b3) ||
        !fill_res_tables<float>(gc.n2, gc.n3, G->h[1], G->h[2], gc.mu, tab, off)) {
        E.tried = true;
        return EQD_OK;
    }
    E.smem = xmarch_smem(gc.n1);
    CUDA_OR_RETURN(cudaFuncSetAttribute((const void *)xmarch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        xmarch_smem(EQD_MAX_N1)));
    const Dense1D M(gc.n1, G->h[0]);
    for (int i = 0; i < gc.n1; ++i) {
        float *r = &rows[(size_t)i * 16];
        for (int o = -3; o <= 3; ++o) {
            const int c = i + o;
            if (c < 0 || c >= gc.n1) continue;
            r[o + 3] = (float)M.d1(i, c);
            r[7 + o + 3] = (float)(gc.mu * M.d2(i, c));
        }
        const int e = std::min(i, gc.n1 - 1 - i);
        r[14] = (float)(-gc.hvol * (e < 4 ? kHw[e].v() : 1.0));
    }
    auto put = [&](DevBuf &b, const void *src, size_t bytes) { return put_table(G, b, src, bytes); };
    CUDA_OR_RETURN(put(E.b2, b2.data(), b2.size() * sizeof(int)));
    CUDA_OR_RETURN(put(E.b3, b3.data(), b3.size() * sizeof(int)));
    CUDA_OR_RETURN(put(E.rows, rows.data(), rows.size() * sizeof(float)));
    CUDA_OR_RETURN(put(E.tab, tab.data(), tab.size() * sizeof(float)));
    CUDA_OR_RETURN(put(E.off, off.data(), off.size() * sizeof(int)));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    XGeom &g = E.g;
    g.n1 = gc.n1;
    g.n2 = gc.n2;
    g.n3 = gc.n3;
    g.n2p = x_row_length(gc.n2);
    g.colstride = x_column(gc.n1, gc.n2, gc.n3);
    g.nt2 = (int)b2.size() - 1;
    g.nt3 = (int)b3.size() - 1;
    g.b2 = E.b2.as<int>();
    g.b3 = E.b3.as<int>();
    g.rows = E.rows.as<float>();
    g.tab = E.tab.as<float>();
    g.off = E.off.as<int>();
    XCoef &C = E.C;
    C.lam = (float)gc.lam;
    C.lpm = (float)(gc.lam + gc.mu);
    C.mu = (float)gc.mu;
    C.mu2 = (float)(2 * gc.mu);
    C.sat = (float)gc.sat_c;
    const double hi = 1.0 / G->h[0];
    C.a = (float)(kD1Int[3].v() * hi);
    C.b = (float)(kD1Int[4].v() * hi);
    C.s0 = (float)(gc.mu * kD2Int[2].v() * hi * hi);
    C.s1 = (float)(gc.mu * kD2Int[3].v() * hi * hi);
    C.s2 = (float)(gc.mu * kD2Int[4].v() * hi * hi);
    for (int k = 0; k < 4; ++k) C.dlo[k] = (float)(kDb[k].v() * hi);
    E.lay = XLayout{gc.n1, gc.n2, gc.n3, g.n2p, gc.PS, gc.colstride, g.colstride};
    // Chunks of 8,192 elements: a column alone at h = 20 m 15.7 ms (17.4 with
    // 16,384, 15.0 with 4,096), 64 columns at h = 25 m 94 ms (93, 98).
    E.nchunks = (int)std::max<long long>(1, (g.colstride + 8191) / 8192);
    E.tried = E.ok = true;
    return EQD_OK;
}

// The tensor map of `cap` columns of x2-fastest vectors: boxes of one x1 plane
// of a tile and its halo, both sides and all components.
static int make_plane_map(const XGeom &g, const float *p, int cap, CUtensorMap &map) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    CUDA_OR_RETURN(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found));
    if (!fn || found != cudaDriverEntryPointSuccess) return fail(EQD_ERR_CUDA, "cuTensorMapEncodeTiled not found");
    const cuuint64_t row = (cuuint64_t)g.n2p * 4;
    const cuuint64_t dims[5] = {(cuuint64_t)g.n2p, (cuuint64_t)g.n3, (cuuint64_t)g.n1, 6, (cuuint64_t)cap};
    const cuuint64_t strides[4] = {row, row * g.n3, row * g.n3 * g.n1, row * g.n3 * g.n1 * 6};
    const cuuint32_t box[5] = {kXR2, kXR3, 1, 6, 1}, one[5] = {1, 1, 1, 1, 1};
    const CUresult r = reinterpret_cast<Encode>(fn)(
        &map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<float *>(p), dims, strides, box, one,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EQD_OK : fail(EQD_ERR_CUDA, "cuTensorMapEncodeTiled: " + std::to_string((int)r));
}

static cudaError_t launch_xmarch(eqd_grid *G, const CUtensorMap &map, float *q, const int8_t *status, double *partials,
                                 int col0, int ncols, cudaStream_t s) {
    const XEngine &E = G->xm;
    const unsigned grid = (unsigned)((long long)ncols * E.g.nt2 * E.g.nt3);
    xmarch_kernel<<<grid, kXThreads, E.smem, s>>>(map, E.g, E.C, q, status, partials, col0, G->err.as<unsigned>());
    return cudaGetLastError();
}

// Layout changes of the flagged columns: x64 += d (fold), or r = src.
static unsigned xlayout_blocks(const XLayout &l, int ncols) {
    return (unsigned)std::min<long long>(kXLayoutBlocks, 6LL * l.n3 * ((l.n2 + 31) / 32) * ncols);
}

static void launch_xfold(eqd_grid *G, double *x64, float *d, const int8_t *status, const int8_t *flag, int ncols,
                         cudaStream_t s) {
    const XLayout &l = G->xm.lay;
    xlayout_kernel<true><<<xlayout_blocks(l, ncols), 256, 0, s>>>(l, x64, d, nullptr, nullptr, status, flag, ncols);
}

static void launch_xresidual(eqd_grid *G, float *r, float *p, float *src, const int8_t *status,
                             const int8_t *flag, int ncols, cudaStream_t s) {
    const XLayout &l = G->xm.lay;
    xlayout_kernel<false><<<xlayout_blocks(l, ncols), 256, 0, s>>>(l, nullptr, r, src, p, status, flag, ncols);
}

static int check_device_error(eqd_grid *G) {
    unsigned h = 0;
    CUDA_OR_RETURN(cudaMemcpyAsync(&h, G->err.p, sizeof(unsigned), cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    if (h != 0) {
        cudaMemsetAsync(G->err.p, 0, sizeof(unsigned), G->stream);
        return fail(EQD_ERR_TIMEOUT, "a device-side bounded wait gave up (error word " + std::to_string(h) + ")");
    }
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Library info
// ---------------------------------------------------------------------------
extern "C" const char *eqd_last_error(void) { return g_last_error.c_str(); }
extern "C" const char *eqd_version(void) { return "eqd-b200 0.1 (sm_100a)"; }

extern "C" void eqd_default_opts(eqd_solve_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->rtol = 1e-10;
    o->atol = 0.0;
    o->itmax = 0;
    o->precond = EQD_PRECOND_NONE;
    o->precision = EQD_PREC_MIXED;
    o->chunk = 0;
    o->reliable_delta = 0.01;
    o->hbm_budget_bytes = 0;
    o->variant = 0;
    o->flags = 0;
}

extern "C" int eqd_device_count(int32_t *count) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) n = 0;
    if (count) *count = n;
    return n > 0 ? EQD_OK : fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
}

// ---------------------------------------------------------------------------
// Grid
// ---------------------------------------------------------------------------
static bool on_node(double x, double l_f, double tol) { return std::fabs(x) <= l_f + tol; }

extern "C" int eqd_grid_create(const eqd_grid_desc *d, eqd_grid **out) {
    if (!d || !out) return fail(EQD_ERR_ARG, "null argument");
    *out = nullptr;
    if (d->order != 4) return fail(EQD_ERR_ARG, "only SBP order 4 (standard_diagonal.toml) is supported");
    if (d->n1 < 9 || d->n2 < 9 || d->n3 < 9)
        return fail(EQD_ERR_ARG, "SBP order 4 needs at least 9 points per axis (got " + std::to_string(d->n1) + "x" +
                                     std::to_string(d->n2) + "x" + std::to_string(d->n3) + ")");
    if (d->n1 > EQD_MAX_N1) return fail(EQD_ERR_ARG, "n1 above the supported maximum of " + std::to_string(EQD_MAX_N1));
    if (!(d->x1_extent > 0) || !(d->x2_hi > d->x2_lo) || !(d->x3_hi > d->x3_lo))
        return fail(EQD_ERR_ARG, "empty domain");
    if (!(d->mu > 0) || !std::isfinite(d->lambda)) return fail(EQD_ERR_ARG, "invalid Lame parameters");
    if (!(d->l_f >= 0)) return fail(EQD_ERR_ARG, "l_f must be non-negative");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
    if (d->device < 0 || d->device >= ndev) return fail(EQD_ERR_ARG, "device ordinal out of range");

    std::unique_ptr<eqd_grid> G(new eqd_grid());
    G->desc = *d;
    GridConst &gc = G->gc;
    gc.n1 = d->n1;
    gc.n2 = d->n2;
    gc.n3 = d->n3;
    G->h[0] = d->x1_extent / (d->n1 - 1);
    G->h[1] = (d->x2_hi - d->x2_lo) / (d->n2 - 1);
    G->h[2] = (d->x3_hi - d->x3_lo) / (d->n3 - 1);
    gc.PS = (d->n1 * d->n2 + 3) / 4 * 4;
    gc.colstride = 6LL * d->n3 * gc.PS;
    gc.lam = d->lambda;
    gc.mu = d->mu;
    gc.hvol = G->h[0] * G->h[1] * G->h[2];
    gc.sat_c = 0.5 / (G->h[0] * kHw[0].v());

    // Omega_f (src/FaultResponse.jl:112-126): |x| <= l_f + 1e-9 max(l_f, 1),
    // and the extreme selected nodes must sit on -l_f and +l_f.
    const double tol = 1e-9 * std::max(d->l_f, 1.0);
    auto select = [&](int n, double lo, double hi, const char *name, int &i0, int &cnt, std::vector<double> &ax) -> int {
        std::vector<double> x(n);
        for (int i = 0; i < n; ++i) x[i] = (i == n - 1) ? hi : lo + (hi - lo) * i / (n - 1);
        i0 = -1;
        cnt = 0;
        for (int i = 0; i < n; ++i)
            if (on_node(x[i], d->l_f, tol)) {
                if (i0 < 0) i0 = i;
                ++cnt;
            }
        if (cnt == 0) return fail(EQD_ERR_ARG, "no fault nodes inside Omega_f");
        if (!(std::fabs(x[i0] + d->l_f) <= tol && std::fabs(x[i0 + cnt - 1] - d->l_f) <= tol))
            return fail(EQD_ERR_ARG, std::string("the elastic grid has no nodes exactly on ") + name +
                                         " = +-l_f; pick a spacing that divides l_f");
        ax.assign(x.begin() + i0, x.begin() + i0 + cnt);
        return EQD_OK;
    };
    int rc = select(d->n2, d->x2_lo, d->x2_hi, "x2", gc.i2f0, gc.n2f, G->x2f);
    if (rc) return rc;
    rc = select(d->n3, d->x3_lo, d->x3_hi, "x3", gc.i3f0, gc.n3f, G->x3f);
    if (rc) return rc;
    gc.nf = gc.n2f * gc.n3f;

    CUDA_OR_RETURN(cudaSetDevice(d->device));  // launch limits below are queried for this device
    fill_op<float>(G->c32, gc, G->h);
    fill_op<double>(G->c64, gc, G->h);
    std::string why;
    if (!make_march_cfg<float>(gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, kMaxT32, 0, gc, G->m32, why))
        return fail(EQD_ERR_ARG, why);
    // FP64: the 384-thread instance where a tile fits, else the 512-thread one.
    G->m64_maxt = kMaxT64;
    if (!make_march_cfg<double>(gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, kMaxT64, 0, gc, G->m64, why)) {
        G->m64_maxt = kMaxT64b;
        if (!make_march_cfg<double>(gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, kMaxT64b, 0, gc, G->m64, why))
            return fail(EQD_ERR_ARG, why);
    }
    // FP32 A-apply variants: one large CTA per SM (640-thread bound, may
    // spill), one CTA of up to 512 threads (no spill), CTAs of up to 256
    // threads so that two share an SM, two columns per thread, and small
    // edge-partitioned tiles (closure rows and interior rows in different CTAs).
    {
        // thread limit, kernel launch bound, columns per thread, tile rows
        // (0: as many as fit), edge partition
        const int lim[kFirstRingVariant] = {kMaxT32, kMaxT32b, 256, kMaxT32c, 192, kMaxT32b, kMaxT32b, 192, 448};
        const int mt[kFirstRingVariant] = {kMaxT32, kMaxT32b, kMaxT32b, kMaxT32c, kMaxT32c, kMaxT32b, kMaxT32b,
                                           kMaxT32b, kMaxT32b};
        const int ln[kFirstRingVariant] = {1, 1, 1, 2, 2, 1, 1, 1, 1};
        const int rows[kFirstRingVariant] = {0, 0, 0, 0, 0, 7, 10, 0, 0};
        const bool edg[kFirstRingVariant] = {false, false, false, false, false, true, true, false, false};
        for (int v = 0; v < kNumVariants; ++v) {
            bool ok;
            if (v < kFirstRingVariant) {
                G->v32_maxt[v] = mt[v];
                G->v32_lanes[v] = ln[v];
                ok = make_march_cfg<float>(gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, lim[v], rows[v], gc, G->v32[v],
                                           why, ln[v], mt[v], edg[v]);
            } else {
                // Ring-march variants: the BP8 lines (n1 = 9, 21, 33) only.
                G->v32_maxt[v] = 0;
                G->v32_lanes[v] = 1;
                ok = make_ring_cfg(gc, G->h, v - kFirstRingVariant, G->v32[v], why);
            }
            if (!ok) {
                G->v32[v] = G->m32;  // fall back to the generic configuration
                G->v32_maxt[v] = kMaxT32;
                G->v32_lanes[v] = 1;
            }
        }
        G->sel32 = 1;
    }
    // Chunks of 8,192 elements in the vector kernels: one FP64 column at 25^3 20.0
    // ms (22.5 with 16,384; 17.5 with 4,096), 64 at h = 40 m 132 (130; 135).
    G->nchunks = (int)std::max<long long>(1, (gc.colstride + 8191) / 8192);

    CUDA_OR_RETURN(cudaSetDevice(d->device));
    {
        int optin = 0;
        CUDA_OR_RETURN(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, d->device));
        size_t need = std::max(G->m32.smem, G->m64.smem);
        for (int v = 0; v < kNumVariants; ++v) need = std::max(need, G->v32[v].smem);
        if ((size_t)optin < need)
            return fail(EQD_ERR_ARG, "stencil tile needs more shared memory than the device offers");
        // A configuration whose second ring does not fit runs the direction
        // update as its own kernel.
        for (MarchCfg *m : {&G->m32, &G->m64})
            if (m->smem_af > (size_t)optin) m->smem_af = 0;
        for (int v = 0; v < kNumVariants; ++v)
            if (G->v32[v].smem_af > (size_t)optin) G->v32[v].smem_af = 0;
        // The limit is a per-kernel attribute shared by every grid of the
        // process: set it to the device maximum, once per device.
        CUDA_OR_RETURN(configure_kernels(optin));
    }
    CUDA_OR_RETURN(cudaDeviceGetAttribute(&G->num_sms, cudaDevAttrMultiProcessorCount, d->device));
    CUDA_OR_RETURN(cudaStreamCreateWithFlags(&G->stream, cudaStreamNonBlocking));
    CUDA_OR_RETURN(cudaStreamCreateWithFlags(&G->stream2, cudaStreamNonBlocking));
    {
        int least = 0, greatest = 0;
        CUDA_OR_RETURN(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream_hi, cudaStreamNonBlocking, greatest));
        CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream2_hi, cudaStreamNonBlocking, greatest));
    }
    CUDA_OR_RETURN(cudaEventCreate(&G->ev0));
    CUDA_OR_RETURN(cudaEventCreate(&G->ev1));
    for (cudaEvent_t *e : {&G->evA, &G->evB, &G->evFork, &G->evJoin, &G->evArest, &G->evBrest})
        CUDA_OR_RETURN(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    CUDA_OR_RETURN(G->err.ensure(sizeof(unsigned)));
    CUDA_OR_RETURN(cudaMemset(G->err.p, 0, sizeof(unsigned)));
    *out = G.release();
    return EQD_OK;
}

extern "C" int eqd_grid_destroy(eqd_grid *G) {
    if (!G) return EQD_OK;
    {
        std::lock_guard<std::mutex> lk(G->mtx);
        if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server; destroy the server first");
    }
    cudaSetDevice(G->desc.device);
    if (G->stream) cudaStreamSynchronize(G->stream);
    if (G->ev0) cudaEventDestroy(G->ev0);
    if (G->ev1) cudaEventDestroy(G->ev1);
    for (cudaEvent_t e : {G->evA, G->evB, G->evFork, G->evJoin, G->evArest, G->evBrest})
        if (e) cudaEventDestroy(e);
    for (cudaStream_t t : {G->stream2, G->stream_hi, G->stream2_hi})
        if (t) cudaStreamDestroy(t);
    if (G->stream) cudaStreamDestroy(G->stream);
    delete G;
    return EQD_OK;
}

extern "C" int eqd_grid_info(const eqd_grid *G, int64_t *ntot, int32_t *nf, int32_t *n2f, int32_t *n3f) {
    if (!G) return fail(EQD_ERR_ARG, "null grid");
    if (ntot) *ntot = 6LL * G->gc.n1 * G->gc.n2 * G->gc.n3;
    if (nf) *nf = G->gc.nf;
    if (n2f) *n2f = G->gc.n2f;
    if (n3f) *n3f = G->gc.n3f;
    return EQD_OK;
}

extern "C" int eqd_grid_fault_axes(const eqd_grid *G, double *x2f, double *x3f) {
    if (!G) return fail(EQD_ERR_ARG, "null grid");
    if (x2f) std::copy(G->x2f.begin(), G->x2f.end(), x2f);
    if (x3f) std::copy(G->x3f.begin(), G->x3f.end(), x3f);
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// eqd_apply (operator hook)
// ---------------------------------------------------------------------------
template <typename T>
static int apply_impl(eqd_grid *G, const double *x, double *y, int ncols, int mode) {
    const GridConst &gc = G->gc;
    const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
    DevBuf hx, dx, dy;
    CUDA_OR_RETURN(hx.ensure(sizeof(double) * ntot * ncols));
    CUDA_OR_RETURN(dx.ensure(sizeof(T) * gc.colstride * ncols));
    CUDA_OR_RETURN(dy.ensure(sizeof(T) * gc.colstride * ncols));
    CUDA_OR_RETURN(cudaMemsetAsync(dx.p, 0, dx.bytes, G->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(hx.p, x, sizeof(double) * ntot * ncols, cudaMemcpyHostToDevice, G->stream));
    const long long nel = ntot * ncols;
    const int tb = 256;
    ref_to_dev_kernel<double, T><<<(unsigned)((nel + tb - 1) / tb), tb, 0, G->stream>>>(
        hx.as<double>(), dx.as<T>(), gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, ncols);
    CUDA_OR_RETURN(cudaGetLastError());
    ColumnSet cs{};
    std::vector<int> neg(ncols, -1), zero(ncols, 0);
    DevBuf sn, sc;
    CUDA_OR_RETURN(sn.ensure(sizeof(int) * ncols));
    CUDA_OR_RETURN(sc.ensure(sizeof(int) * ncols));
    CUDA_OR_RETURN(cudaMemcpyAsync(sn.p, neg.data(), sizeof(int) * ncols, cudaMemcpyHostToDevice, G->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(sc.p, zero.data(), sizeof(int) * ncols, cudaMemcpyHostToDevice, G->stream));
    cs.slip_node = sn.as<int>();
    cs.slip_comp = sc.as<int>();
    if (mode == 0) {
        CUDA_OR_RETURN((launch_march<T, T, MODE_AP>(G, dx.as<T>(), dy.as<T>(), cs, nullptr, ncols)));
    } else if (mode == 2 && sizeof(T) == 4 && G->pin == kXMarchVariant && G->xm.ok) {
        // The x1 march, on x2-fastest copies.
        const XLayout &l = G->xm.lay;
        DevBuf vx, vy;
        CUDA_OR_RETURN(vx.ensure(sizeof(float) * l.cnew * ncols));
        CUDA_OR_RETURN(vy.ensure(sizeof(float) * l.cnew * ncols));
        CUDA_OR_RETURN(cudaMemsetAsync(vx.p, 0, vx.bytes, G->stream));
        CUDA_OR_RETURN(cudaMemsetAsync(vy.p, 0, vy.bytes, G->stream));
        CUtensorMap map;
        int rc = make_plane_map(G->xm.g, vx.as<float>(), ncols, map);
        if (rc) return rc;
        const unsigned nb = (unsigned)((nel + tb - 1) / tb);
        xref_kernel<true><<<nb, tb, 0, G->stream>>>(l, hx.as<double>(), vx.as<float>(), ncols);
        CUDA_OR_RETURN(launch_xmarch(G, map, vy.as<float>(), nullptr, nullptr, 0, ncols, G->stream));
        xref_kernel<false><<<nb, tb, 0, G->stream>>>(l, hx.as<double>(), vy.as<float>(), ncols);
        CUDA_OR_RETURN(cudaGetLastError());
        CUDA_OR_RETURN(cudaMemcpyAsync(y, hx.p, sizeof(double) * nel, cudaMemcpyDeviceToHost, G->stream));
        CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
        return check_device_error(G);
    } else if (mode == 2) {
        DevBuf part;
        int nt = nparts(G->m64);
        for (int v = 0; v < kNumVariants; ++v) nt = std::max(nt, nparts(G->v32[v]));
        CUDA_OR_RETURN(part.ensure(sizeof(double) * 2 * ncols * nt));
        CUDA_OR_RETURN((launch_march<T, T, MODE_A>(G, dx.as<T>(), dy.as<T>(), cs, part.as<double>(), ncols)));
    } else {
        CUDA_OR_RETURN((launch_march<T, T, MODE_RHS>(G, dx.as<T>(), dy.as<T>(), cs, nullptr, ncols)));
    }
    dev_to_ref_kernel<T, double><<<(unsigned)((nel + tb - 1) / tb), tb, 0, G->stream>>>(
        dy.as<T>(), hx.as<double>(), gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, ncols);
    CUDA_OR_RETURN(cudaGetLastError());
    CUDA_OR_RETURN(cudaMemcpyAsync(y, hx.p, sizeof(double) * ntot * ncols, cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    return check_device_error(G);
}

extern "C" int eqd_apply(eqd_grid *G, const double *x, double *y, int32_t ncols, int32_t mode, int32_t precision) {
    if (!G || !x || !y) return fail(EQD_ERR_ARG, "null argument");
    if (ncols < 1) return fail(EQD_ERR_ARG, "ncols must be >= 1");
    if (mode < 0 || mode > 2) return fail(EQD_ERR_ARG, "mode must be 0 (A), 1 (HP_DSAT) or 2 (A, input in range(P))");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    if (precision == EQD_PREC_FP64) return apply_impl<double>(G, x, y, ncols, mode);
    if (precision == EQD_PREC_MIXED) {
        if (G->pin == kXMarchVariant) {
            int rc = ensure_xmarch(G);
            if (rc) return rc;
        }
        return apply_impl<float>(G, x, y, ncols, mode);
    }
    return fail(EQD_ERR_ARG, "unknown precision");
}

// ---------------------------------------------------------------------------
// Autotuning of the FP32 A-apply launch variant (once per grid): each variant
// is timed on `ncols` device-resident columns; the fastest is kept. The
// choice is fixed for the grid's lifetime, so every column of every later
// call uses the same tile partition (and the same reduction order).
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// Batched CG driver
// ---------------------------------------------------------------------------
struct BatchSpec {
    int ncols;
    const int *slip_node;        // host, per column (unit slip), or null
    const int *slip_comp;
    const double *slip_dense;    // host [ncols][2][nf] or null
    const double *rhs;           // host reference-layout RHS [ncols][ntot] (explicit-RHS solve) or null
    double *u_out;               // host reference-layout solution (explicit-RHS solve) or null
    double *kcols;               // host 2nf x ncols output (slip-driven) or null
    double *kdev;                // device 2nf x ncols output (slip-driven) or null
    int32_t *iters;
    int8_t *status;
};

// Whether the options and the pinned variant leave a solve to the on-chip CG.
template <typename T>
static bool allows_resident(const eqd_grid *G, const eqd_solve_opts &o) {
    const int pin = sizeof(T) == 4 ? G->pin : G->pin64;
    return o.precond != EQD_PRECOND_JACOBI && (pin < 0 || pin == kResidentVariant);
}

// What runs a solve's iterations: resident_cg_kernel, or xmarch_kernel on
// x2-fastest vectors, or (neither) the streamed x1-fastest path.
struct Path {
    bool resident = false, xm = false;
};

// `on_chip`: explicit right-hand sides (`gen`) that run resident.
template <typename T>
static int choose_path(eqd_grid *G, const eqd_solve_opts &o, bool gen, bool on_chip, Path &p) {
    p = Path{};
    p.resident = gen && on_chip;
    if (!gen && allows_resident<T>(G, o)) {
        ResEngine &E = sizeof(T) == 4 ? G->res32 : G->res64;
        int rc = ensure_resident<T>(G, E);
        if (rc) return rc;
        p.resident = E.ok && !E.few;
    }
    if (sizeof(T) == 4 && !gen && !p.resident && o.precond != EQD_PRECOND_JACOBI &&
        (G->pin < 0 || G->pin == kResidentVariant || G->pin == kXMarchVariant)) {
        int rc = ensure_xmarch(G);
        if (rc) return rc;
        p.xm = G->xm.ok;
    }
    return EQD_OK;
}

// Device bytes of a slot: x in FP64; r, p, q (mixed: and d) in the working
// precision, and the second direction buffer where the direction update is fused
// into the apply; the x1 march's vectors with padded x2 lines.
template <typename T>
static size_t slot_bytes(const eqd_grid *G, const eqd_solve_opts &o, bool gen, const Path &p) {
    const GridConst &gc = G->gc;
    const bool fused = !p.resident && !p.xm && !gen && o.precond != EQD_PRECOND_JACOBI && (o.flags & EQD_FLAG_FUSE);
    const size_t nvec = 3 + (sizeof(T) == 4 ? 1 : 0) + (fused ? 1 : 0);
    const size_t vec = p.xm ? (size_t)x_column(gc.n1, gc.n2, gc.n3) : (size_t)gc.colstride;
    return (size_t)gc.colstride * 8 + vec * nvec * sizeof(T) + (size_t)16 * gc.nf + 1024;
}

// The slots of a solve of `ncols` columns, and the path that they run on.
template <typename T>
static int resolve_chunk(eqd_grid *G, const eqd_solve_opts &o, int ncols, bool gen, bool on_chip, Path &path, int &chunk) {
    int rc = choose_path<T>(G, o, gen, on_chip, path);
    if (rc) return rc;
    size_t budget = o.hbm_budget_bytes;
    if (budget == 0) {
        size_t fr = 0, tot = 0;
        CUDA_OR_RETURN(cudaMemGetInfo(&fr, &tot));
        const size_t keep = (size_t)2 << 30;
        budget = fr > keep ? fr - keep : fr / 2;
    }
    // (A budget that only the padding overdraws streams x1-fastest.)
    if (path.xm && budget < slot_bytes<T>(G, o, gen, path)) path.xm = false;
    long long cap = (long long)(budget / slot_bytes<T>(G, o, gen, path));
    if (cap < 1) return fail(EQD_ERR_OOM, "HBM budget too small for one column");
    const long long want =
        o.chunk > 0 ? o.chunk : ((G->chunk_tuned > 0 && sizeof(T) == 4) ? G->chunk_tuned : cap);
    chunk = (int)std::min<long long>(want, ncols);
    if ((long long)chunk > cap) chunk = (int)cap;
    return EQD_OK;
}

// Columns [c0, c0 + n) of the slot arrays, recorded on stream `s`: every
// pointer is offset to the span, so two spans are independent CG batches.
struct Span {
    int c0, n;
    cudaStream_t s;
    bool split;  // one of two halves whose kernels overlap
};

template <typename T>
struct IterPtrs {
    ColumnSet cs;
    ColState st;
    T *r, *p, *q;
    T *p2;  // fused direction update: the other direction buffer
    float *d;
    double *x64, *apply_part, *res_part, *rr_part;
};

template <typename T>
static IterPtrs<T> span_ptrs(eqd_grid *G, Workspace &W, const SolveParams &sp, const ColState &st0, const Span &sp_) {
    const GridConst &gc = G->gc;
    const long long c0 = sp_.c0;
    IterPtrs<T> P{};
    P.cs.ncols = sp_.n;
    P.cs.slip_node = W.slip_node.as<int>() + c0;
    P.cs.slip_comp = W.slip_comp.as<int>() + c0;
    P.cs.slip_dense = W.slip_dense.p ? W.slip_dense.as<double>() + c0 * 2 * gc.nf : nullptr;
    P.cs.status = W.status.as<int8_t>() + c0;
    P.st = ColState{st0.gamma + c0, st0.beta + c0, st0.rr_ref + c0, st0.tol + c0, st0.bnorm + c0,
                    st0.iters + c0, st0.status + c0, st0.flag + c0, st0.pp + c0};
    P.r = W.v0.as<T>() + c0 * sp.colstride;
    P.p = W.v1.as<T>() + c0 * sp.colstride;
    P.q = W.v2.as<T>() + c0 * sp.colstride;
    P.p2 = W.v4.p ? W.v4.as<T>() + c0 * gc.colstride : nullptr;
    P.d = W.v3.p ? W.v3.as<float>() + c0 * sp.colstride : nullptr;
    P.x64 = W.x64.as<double>() + c0 * gc.colstride;
    P.apply_part = W.apply_part.as<double>() + c0 * sp.ntiles * 2;
    P.res_part = W.res_part.as<double>() + c0 * nparts(G->m64) * 2;
    P.rr_part = W.rr_part.as<double>() + c0 * sp.nchunks * 2;
    return P;
}

// The direction of iteration k when the direction update is fused into the
// apply: iteration k reads the previous direction from one buffer and writes
// the new one to the other (v1 at even k, v4 at odd k; kIter is even, so a
// graph launch always starts with the current direction in v1).
template <typename T>
static T *dir_in(const IterPtrs<T> &P, int k) { return (k & 1) ? P.p2 : P.p; }
template <typename T>
static T *dir_out(const IterPtrs<T> &P, int k) { return (k & 1) ? P.p : P.p2; }

// Returns a launch's error from a function of CUDA errors.
#define EQD_TRY(call)                                \
    do {                                             \
        const cudaError_t try_e = (call);            \
        if (try_e != cudaSuccess) return try_e;      \
    } while (0)

// A pending eqd_test_inject_failure: the launch is not made.
static bool injected_launch_error(eqd_grid *G) {
    const bool f = G->test_fail_launch;
    G->test_fail_launch = false;
    return f;
}

// The stencil apply of CG iteration k (q = A p, partial p.q); fused: with
// p = r + beta p formed on the way in.
template <typename T>
static cudaError_t record_apply(eqd_grid *G, Workspace &W, int generic, int fused, int k, const SolveParams &sp,
                         const ColState &st0, const Span &sn) {
    IterPtrs<T> P = span_ptrs<T>(G, W, sp, st0, sn);
    if (injected_launch_error(G)) return cudaErrorLaunchOutOfResources;
    if (sp.xlayout) return launch_xmarch(G, W.pmap, (float *)P.q, P.cs.status, P.apply_part, sn.c0, sn.n, sn.s);
    if (generic) return launch_march<T, T, MODE_AP>(G, P.p, P.q, P.cs, P.apply_part, sn.n, -1, sn.s);
    if (fused) {
        ColumnSet cs = P.cs;
        cs.pold = dir_in(P, k);
        cs.pnew = dir_out(P, k);
        cs.beta = P.st.beta;
        return launch_march<T, T, MODE_AF>(G, P.r, P.q, cs, P.apply_part, sn.n, -1, sn.s);
    }
    return launch_march<T, T, MODE_A>(G, P.p, P.q, P.cs, P.apply_part, sn.n, -1, sn.s);
}

// CTA size of the vector kernels inside the iterations: small enough to fit
// beside resident stencil CTAs on an SM (the update kernel's 128 threads x
// 62-70 registers take the 8 K registers that two 224-thread, 128-register
// stencil CTAs leave free), so the other half's updates can run while an
// apply is in flight.
static constexpr int kVecThreads = 128;
// With a split batch the vector kernels run on 4 CTAs per SM (grid-stride):
// they fit beside the other half's stencil CTAs and still stream at close to
// HBM speed (measured at h = 50 m: 1, 2, 4, 8 CTAs per SM and one CTA per item
// gave 6.0, 6.6, 6.5, 6.3 k columns/s; one chain with one CTA per item 6.2 k).
static constexpr int kVecCtasPerSm = 4;

// Mixed precision: the flagged columns' FP64 true residual.
template <typename T>
static cudaError_t record_reliable(eqd_grid *G, const IterPtrs<T> &P, const SolveParams &sp, const Span &sn) {
    // One CTA per item: in most iterations no column is flagged and every
    // CTA returns at once.
    const unsigned items = (unsigned)((long long)sn.n * G->nchunks);
    if (sp.xlayout) launch_xfold(G, P.x64, P.d, P.st.status, P.st.flag, sn.n, sn.s);
    else fold_correction_kernel<<<items, kVecThreads, 0, sn.s>>>(P.x64, P.d, P.st, sp, sn.n);
    ColumnSet cf = P.cs;
    cf.flag = P.st.flag;
    cf.dinv = sp.precond ? G->dinv64.as<double>() : nullptr;
    EQD_TRY(cudaGetLastError());
    // (x2-fastest vectors: q is read by now, and holds the residuals until r has them.)
    EQD_TRY((launch_march<double, float, MODE_RHS>(G, P.x64, sp.xlayout ? (float *)P.q : (float *)P.r, cf, P.res_part,
                                                   sn.n, -1, sn.s)));
    if (sp.xlayout)
        launch_xresidual(G, (float *)P.r, (float *)P.p, (float *)P.q, P.st.status, P.st.flag, sn.n, sn.s);
    SolveParams sp2 = sp;
    sp2.ntiles = nparts(G->m64);
    cg_true_residual_kernel<<<(unsigned)((sn.n + 3) / 4), 128, 0, sn.s>>>(P.st, sp2, P.res_part, sn.n, 1);
    return cudaGetLastError();
}

// The rest of iteration k: x, r updates; scalars; reliable update (mixed);
// the next direction (unless the next apply forms it).
template <typename T>
static cudaError_t record_rest(eqd_grid *G, Workspace &W, int mixed, int fused, int k, const SolveParams &sp,
                        const ColState &st0, const Span &sn) {
    IterPtrs<T> P = span_ptrs<T>(G, W, sp, st0, sn);
    const T *pk = fused ? dir_out(P, k) : P.p;  // this iteration's direction
    const int nch = sp.nchunks;
    const double *dinv64 = sp.precond ? G->dinv64.as<double>() : nullptr;
    const float *dinv32 = sp.precond ? G->dinv32.as<float>() : nullptr;
    // Split: a few CTAs per SM (grid-stride over the items) so they fit
    // beside the other half's stencil CTAs; one chain: one CTA per item.
    const long long items = (long long)sn.n * nch;
    const unsigned nb = (unsigned)(sn.split ? std::min<long long>(items, (long long)G->num_sms * kVecCtasPerSm) : items);
    // Mixed precision: the bulk-staged vector kernels (measured at h = 50 m,
    // 2,178 columns: 7,213 vs 6,771 columns/s with the register versions).
    // FP64: the register versions (the bulk-staged ones measured 17 % slower
    // beside the FP64 stencil).
    unsigned *err = G->err.as<unsigned>();
    const unsigned sb = (unsigned)((sn.n + 3) / 4);
    if (sp.xlayout) {
        cg_step_bulk_kernel<<<nb, kVecThreads, kStepBulkSmem, sn.s>>>(P.d, (float *)P.r, (float *)P.p, (const float *)P.q,
                                                                      P.apply_part, P.st, sp, P.rr_part, sn.n, err);
        cg_check_kernel<<<sb, 128, 0, sn.s>>>(P.st, sp, P.apply_part, P.rr_part, sn.n);
        EQD_TRY(cudaGetLastError());
        return record_reliable<T>(G, P, sp, sn);
    }
    if (mixed) {
        cg_update_bulk_kernel<float, float><<<nb, kVecThreads, kUpdateBulkSmem, sn.s>>>(
            P.d, (float *)P.r, (const float *)pk, (const float *)P.q, P.apply_part, P.st, sp, P.rr_part, dinv32, sn.n,
            err);
    } else {
        cg_update_kernel<double, double><<<nb, kVecThreads, 0, sn.s>>>(P.x64, (double *)P.r, (const double *)pk,
                                                              (const double *)P.q, P.apply_part, P.st, sp,
                                                              P.rr_part, dinv64, sn.n);
    }
    cg_scalar_kernel<<<sb, 128, 0, sn.s>>>(P.st, sp, P.apply_part, P.rr_part, sn.n, mixed);
    EQD_TRY(cudaGetLastError());
    if (mixed) EQD_TRY(record_reliable<T>(G, P, sp, sn));
    if (!fused) {
        const T *dinvT = (const T *)(sizeof(T) == 4 ? (const void *)dinv32 : (const void *)dinv64);
        if (mixed)
            cg_pupdate_bulk_kernel<T><<<nb, kVecThreads, kDirBulkSmem, sn.s>>>(P.p, P.r, P.st, sp, dinvT, sn.n, err);
        else
            cg_pupdate_kernel<T><<<nb, kVecThreads, 0, sn.s>>>(P.p, P.r, P.st, sp, nullptr, dinvT, sn.n);
    }
    return cudaGetLastError();
}

// Capture kIter CG iterations over `cap` slots. Large batches are split in
// two halves on two streams whose stencil applies alternate: the
// arithmetic-bound apply of one half runs while the memory-bound vector
// updates of the other half stream through HBM.
template <typename T>
static cudaError_t record_iterations(eqd_grid *G, Workspace &W, int cap, int mixed, int generic, int fused,
                              const SolveParams &sp, const ColState &st, int kIter, bool split) {
    if (!split) {
        const Span all{0, cap, G->stream, false};
        for (int k = 0; k < kIter; ++k) {
            EQD_TRY(record_apply<T>(G, W, generic, fused, k, sp, st, all));
            EQD_TRY(record_rest<T>(G, W, mixed, fused, k, sp, st, all));
        }
        return cudaSuccess;
    }
    // Applies on normal-priority streams, the rest of each iteration on
    // high-priority streams (node priorities are kept at instantiation), so
    // that freed SM slots go to the short memory-bound kernels first.
    const int h0 = cap / 2;
    const Span A{0, h0, G->stream, true}, B{h0, cap - h0, G->stream2, true};
    const Span Ah{0, h0, G->stream_hi, true}, Bh{h0, cap - h0, G->stream2_hi, true};
    EQD_TRY(cudaEventRecord(G->evFork, A.s));
    for (cudaStream_t t : {B.s, Ah.s, Bh.s}) EQD_TRY(cudaStreamWaitEvent(t, G->evFork, 0));
    for (int k = 0; k < kIter; ++k) {
        if (k > 0) {
            EQD_TRY(cudaStreamWaitEvent(A.s, G->evB, 0));      // B's previous apply is done
            EQD_TRY(cudaStreamWaitEvent(A.s, G->evArest, 0));  // A's previous direction is ready
        }
        EQD_TRY(record_apply<T>(G, W, generic, fused, k, sp, st, A));
        EQD_TRY(cudaEventRecord(G->evA, A.s));
        EQD_TRY(cudaStreamWaitEvent(B.s, G->evA, 0));          // B's apply follows A's
        if (k > 0) EQD_TRY(cudaStreamWaitEvent(B.s, G->evBrest, 0));
        EQD_TRY(record_apply<T>(G, W, generic, fused, k, sp, st, B));
        EQD_TRY(cudaEventRecord(G->evB, B.s));
        EQD_TRY(cudaStreamWaitEvent(Ah.s, G->evA, 0));
        EQD_TRY(record_rest<T>(G, W, mixed, fused, k, sp, st, Ah));
        EQD_TRY(cudaEventRecord(G->evArest, Ah.s));
        EQD_TRY(cudaStreamWaitEvent(Bh.s, G->evB, 0));
        EQD_TRY(record_rest<T>(G, W, mixed, fused, k, sp, st, Bh));
        EQD_TRY(cudaEventRecord(G->evBrest, Bh.s));
    }
    EQD_TRY(cudaEventRecord(G->evJoin, B.s));
    EQD_TRY(cudaStreamWaitEvent(A.s, G->evJoin, 0));
    EQD_TRY(cudaStreamWaitEvent(A.s, G->evArest, 0));
    EQD_TRY(cudaStreamWaitEvent(A.s, G->evBrest, 0));
    return cudaSuccess;
}

// Resident iterations of `cap` slots: every active column runs until it needs
// its true residual (mixed) or is done, at most kmax iterations, `rounds`
// times.
template <typename T>
static cudaError_t record_resident(eqd_grid *G, Workspace &W, int cap, int mixed, const SolveParams &sp, const ColState &st,
                            int kmax, int rounds) {
    const Span all{0, cap, G->stream, false};
    IterPtrs<T> P = span_ptrs<T>(G, W, sp, st, all);
    T *x = sizeof(T) == 4 ? (T *)P.d : (T *)P.x64;
    for (int k = 0; k < rounds; ++k) {
        if (injected_launch_error(G)) return cudaErrorLaunchOutOfResources;
        EQD_TRY(launch_resident<T>(G, sizeof(T) == 4 ? G->res32 : G->res64, x, P.r, P.p, P.st, sp, mixed, kmax, cap,
                                   G->stream));
        if (mixed) EQD_TRY(record_reliable<T>(G, P, sp, all));
    }
    return cudaSuccess;
}

// Jacobi weights dinv = 1 / diag(A) (zeros floored to 1), computed once per
// grid; a negative diagonal entry is an error, as in the reference.
static int ensure_jacobi(eqd_grid *G) {
    if (G->jacobi_ready) return EQD_OK;
    const GridConst &gc = G->gc;
    CUDA_OR_RETURN(G->dinv64.ensure(sizeof(double) * gc.colstride));
    CUDA_OR_RETURN(G->dinv32.ensure(sizeof(float) * gc.colstride));
    CUDA_OR_RETURN(cudaMemsetAsync(G->dinv64.p, 0, sizeof(double) * gc.colstride, G->stream));
    CUDA_OR_RETURN(cudaMemsetAsync(G->dinv32.p, 0, sizeof(float) * gc.colstride, G->stream));
    DevBuf neg;
    CUDA_OR_RETURN(neg.ensure(sizeof(unsigned)));
    CUDA_OR_RETURN(cudaMemsetAsync(neg.p, 0, sizeof(unsigned), G->stream));
    const long long n = 6LL * gc.n1 * gc.n2 * gc.n3;
    jacobi_diag_kernel<<<(unsigned)((n + 255) / 256), 256, 0, G->stream>>>(
        G->c64, gc.n1, gc.n2, gc.n3, gc.PS, nullptr, G->dinv64.as<double>(), G->dinv32.as<float>(), neg.as<unsigned>());
    CUDA_OR_RETURN(cudaGetLastError());
    unsigned h = 0;
    CUDA_OR_RETURN(cudaMemcpyAsync(&h, neg.p, sizeof(unsigned), cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    if (h) return fail(EQD_ERR_ARG, "diag(A) has negative entries; A is not PSD and a Jacobi preconditioner "
                                    "would not be SPD");
    G->jacobi_ready = true;
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Slot engine: a fixed set of column slots, each holding one right-hand side's
// CG state. A column enters a free slot (its vectors are zeroed and r0 = b is
// evaluated for it alone), runs with every other occupied slot in the
// graph-captured iterations, and leaves when its status is final; its slot is
// then free for the next column. A column's arithmetic does not depend on the
// other slots (every reduction is per column, in a fixed order), so a column
// gives the same bits whenever and beside whatever it runs.
// ---------------------------------------------------------------------------
struct ColWork {
    int slip_node = -1;                  // unit slip at this Omega_f node (-1: none)
    int slip_comp = 0;                   // 0 -> s2, 1 -> s3
    const double *slip_dense = nullptr;  // host [2][nf] slip field, or null
    const double *rhs = nullptr;         // host reference-layout right-hand side (explicit-RHS solve), or null
    long long tag = 0;                   // the caller's id for the column
};

struct ColDone {
    long long tag;
    int slot;
    int iters;
    int8_t status;
};

static int tune_by_iterations(eqd_grid *G, const eqd_solve_opts &o, int ncols, bool with_resident = false);

template <typename T>
struct SlotRun {
    eqd_grid *G = nullptr;
    Workspace *W = nullptr;
    int cap = 0, mixed = 0, generic = 0, dense = 0;
    int fused = 0;  // the direction update runs inside the stencil apply (MODE_AF)
    int resident = 0;            // iterations run in resident_cg_kernel
    int xm = 0;                  // the FP32 vectors are x2-fastest (xmarch_kernel)
    int kmax = 256, rounds = 1;  // resident: iterations a launch may run, launches per graph
    long long itmax = 0;
    SolveParams sp{};
    ColState st{};
    std::vector<int> hn, hc, hslot, hdst;
    std::vector<int> seen;  // a slot's iterations at the last collect()
    std::vector<int8_t> hnew;
    PinnedArr<int> hit;     // per-slot iteration counts (read back every graph launch)
    PinnedArr<int8_t> hst;  // per-slot status
    std::vector<long long> tag;  // -1: free slot
    int held = 0;                // occupied slots (running or finished, not yet released)
    int64_t launches = 0;
    static constexpr int kIter = 10;

    // `tuning`: the caller times kIter iterations a launch.
    int setup(eqd_grid *g, const eqd_solve_opts &o, int capacity, bool gen, bool dns, const Path &path,
              bool tuning = false) {
        G = g;
        W = &G->ws;
        cap = capacity;
        mixed = o.precision == EQD_PREC_MIXED;
        generic = gen;
        dense = dns;
        const GridConst &gc = G->gc;
        const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
        resident = path.resident;
        xm = path.xm;
        kmax = tuning ? kIter : 256;
        rounds = mixed && !tuning ? 2 : 1;
        if (mixed && !G->tuned && !resident && !xm) {
            int rc = tune_by_iterations(G, o, std::min(cap, 1024));
            if (rc) return rc;
        }
        const int nt32 = nparts(G->v32[G->sel32]), nt64 = nparts(G->m64);
        Workspace &w = *W;
        const size_t vec64 = (size_t)gc.colstride * cap, vec = xm ? (size_t)G->xm.g.colstride * cap : vec64;
        CUDA_OR_RETURN(w.x64.ensure(sizeof(double) * vec64));
        CUDA_OR_RETURN(w.v0.ensure(sizeof(T) * vec));
        CUDA_OR_RETURN(w.v1.ensure(sizeof(T) * vec));
        CUDA_OR_RETURN(w.v2.ensure(sizeof(T) * vec));
        if (mixed) CUDA_OR_RETURN(w.v3.ensure(sizeof(float) * vec));
        {
            const MarchCfg &mc = sizeof(T) == 4 ? G->v32[G->sel32] : G->m64;
            fused = !resident && !xm && !generic && o.precond != EQD_PRECOND_JACOBI && (o.flags & EQD_FLAG_FUSE) && mc.smem_af > 0;
        }
        if (fused) CUDA_OR_RETURN(w.v4.ensure(sizeof(T) * vec64));
        else w.v4.release();
        int ntmax = std::max(nt64, nparts(G->m32));
        for (int v = 0; v < kNumVariants; ++v) ntmax = std::max(ntmax, nparts(G->v32[v]));
        if (xm) ntmax = std::max(ntmax, G->xm.g.nt2 * G->xm.g.nt3);
        CUDA_OR_RETURN(w.apply_part.ensure(sizeof(double) * 2 * cap * ntmax));
        CUDA_OR_RETURN(w.res_part.ensure(sizeof(double) * 2 * cap * std::max(nt64, G->nchunks)));
        const int nch = xm ? G->xm.nchunks : G->nchunks;
        CUDA_OR_RETURN(w.rr_part.ensure(sizeof(double) * 2 * cap * nch));
        for (DevBuf *b : {&w.gamma, &w.beta, &w.rr_ref, &w.tol, &w.bnorm, &w.pp}) CUDA_OR_RETURN(b->ensure(sizeof(double) * cap));
        CUDA_OR_RETURN(w.iters.ensure(sizeof(int) * cap));
        CUDA_OR_RETURN(w.status.ensure(cap));
        CUDA_OR_RETURN(w.flag.ensure(cap));
        CUDA_OR_RETURN(w.newmask.ensure(cap));
        CUDA_OR_RETURN(w.slot_list.ensure(sizeof(int) * cap));
        CUDA_OR_RETURN(w.dst_list.ensure(sizeof(int) * cap));
        CUDA_OR_RETURN(w.slip_node.ensure(sizeof(int) * cap));
        CUDA_OR_RETURN(w.slip_comp.ensure(sizeof(int) * cap));
        if (dense) CUDA_OR_RETURN(w.slip_dense.ensure(sizeof(double) * 2 * gc.nf * cap));
        else w.slip_dense.release();
        CUDA_OR_RETURN(w.kout.ensure(sizeof(double) * 2 * gc.nf * cap));
        if (generic) CUDA_OR_RETURN(w.hbuf.ensure(sizeof(double) * ntot * cap));

        st = ColState{w.gamma.as<double>(), w.beta.as<double>(), w.rr_ref.as<double>(), w.tol.as<double>(),
                      w.bnorm.as<double>(), w.iters.as<int>(), w.status.as<int8_t>(), w.flag.as<int8_t>(), w.pp.as<double>()};
        sp = SolveParams{};
        sp.rtol = o.rtol;
        sp.atol = o.atol;
        sp.itmax = o.itmax;
        sp.delta = o.reliable_delta > 0 ? o.reliable_delta : 0.01;
        sp.ntiles = xm ? G->xm.g.nt2 * G->xm.g.nt3 : sizeof(T) == 4 ? nt32 : nt64;
        sp.nchunks = nch;
        sp.colstride = xm ? G->xm.g.colstride : gc.colstride;
        sp.xlayout = xm;
        if (xm) {
            int rc = make_plane_map(G->xm.g, w.v1.as<float>(), cap, w.pmap);
            if (rc) return rc;
        }
        sp.ntot = ntot;
        sp.precond = o.precond == EQD_PRECOND_JACOBI;
        if (sp.precond) {
            int rc = ensure_jacobi(G);
            if (rc) return rc;
        }
        itmax = o.itmax > 0 ? o.itmax : 2 * ntot;

        // Every slot starts free: status IDLE everywhere, vectors zeroed as
        // columns enter.
        hn.assign(cap, -1);
        hc.assign(cap, 0);
        CUDA_OR_RETURN(hit.assign(cap, 0));
        CUDA_OR_RETURN(hst.assign(cap, (int8_t)COL_IDLE));
        hnew.assign(cap, 0);
        seen.assign(cap, 0);
        tag.assign(cap, -1);
        hslot.resize(cap);
        hdst.resize(cap);
        held = 0;
        CUDA_OR_RETURN(cudaMemcpyAsync(w.status.p, hst.data(), cap, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemsetAsync(w.flag.p, 0, cap, G->stream));

        // Graph of kIter iterations over all slots, captured once per
        // (capacity, precision, mode, launch variant, preconditioner, split).
        const bool split = cap >= 64 && !(o.flags & EQD_FLAG_NO_SPLIT);
        // Everything the captured kernels bake in: sizes, options and every
        // workspace pointer (a buffer that grew or was released since the
        // capture must not be reached through the old graph).
        std::vector<uint64_t> kv = {(uint64_t)cap, (uint64_t)o.precision, (uint64_t)generic, (uint64_t)G->sel32,
                                    (uint64_t)o.precond, (uint64_t)split, (uint64_t)sp.itmax, (uint64_t)fused, (uint64_t)resident,
                                    (uint64_t)(kmax * 16 + rounds), (uint64_t)xm};
        for (double d : {sp.rtol, sp.atol, sp.delta}) {
            uint64_t b;
            std::memcpy(&b, &d, sizeof(b));
            kv.push_back(b);
        }
        for (const void *q : {w.x64.p, w.v0.p, w.v1.p, w.v2.p, w.v3.p, w.v4.p, w.apply_part.p, w.res_part.p, w.rr_part.p,
                              w.gamma.p, w.beta.p, w.rr_ref.p, w.tol.p, w.bnorm.p, w.pp.p, w.iters.p, w.status.p, w.flag.p,
                              w.slip_node.p, w.slip_comp.p, w.slip_dense.p, G->dinv64.p, G->dinv32.p})
            kv.push_back((uint64_t)(uintptr_t)q);
        if (!w.graph || w.graph_key != kv) {
            if (w.graph) cudaGraphExecDestroy(w.graph);
            w.graph = nullptr;
            w.graph_key.clear();
            cudaGraph_t g = nullptr;
            cudaGetLastError();  // (an earlier call's, already reported)
            CUDA_OR_RETURN(cudaStreamBeginCapture(G->stream, cudaStreamCaptureModeThreadLocal));
            const cudaError_t re = resident
                                       ? record_resident<T>(G, w, cap, mixed, sp, st, kmax, rounds)
                                       : record_iterations<T>(G, w, cap, mixed, generic, fused, sp, st, kIter, split);
            cudaError_t ce = cudaStreamEndCapture(G->stream, &g);
            if (re != cudaSuccess) {  // a graph without one of its kernels must not run
                if (g) cudaGraphDestroy(g);
                cudaGetLastError();
                return fail(EQD_ERR_CUDA, std::string("recording the CG iterations: ") + cudaGetErrorString(re));
            }
            if (ce != cudaSuccess) return fail(EQD_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
            ce = cudaGraphInstantiate(&w.graph, g, cudaGraphInstantiateFlagUseNodePriority);
            cudaGraphDestroy(g);
            if (ce != cudaSuccess) return fail(EQD_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ce));
            w.graph_key = kv;
            w.graph_iters = kIter;
            w.graph_split = split;
        }
        return EQD_OK;
    }

    int free_slots() const { return cap - held; }

    ColumnSet colset() const {
        ColumnSet cs{};
        cs.ncols = cap;
        cs.slip_node = W->slip_node.as<int>();
        cs.slip_comp = W->slip_comp.as<int>();
        cs.slip_dense = dense ? W->slip_dense.as<double>() : nullptr;
        cs.status = W->status.as<int8_t>();
        return cs;
    }

    // Put up to n columns into free slots and evaluate their r0 = b; `taken`
    // is how many entered.
    int admit(const ColWork *work, int n, int &taken) {
        taken = 0;
        const GridConst &gc = G->gc;
        const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
        Workspace &w = *W;
        std::fill(hnew.begin(), hnew.end(), (int8_t)0);
        for (int s = 0; s < cap && taken < n; ++s) {
            if (tag[s] >= 0) continue;
            const ColWork &c = work[taken++];
            tag[s] = c.tag;
            hn[s] = c.slip_node;
            hc[s] = c.slip_comp;
            hst[s] = COL_ACTIVE;
            hit[s] = seen[s] = 0;
            hnew[s] = 1;
            ++held;
            if (dense) {
                if (c.slip_dense)
                    CUDA_OR_RETURN(cudaMemcpyAsync(w.slip_dense.as<double>() + (size_t)s * 2 * gc.nf, c.slip_dense,
                                                   sizeof(double) * 2 * gc.nf, cudaMemcpyHostToDevice, G->stream));
                else
                    CUDA_OR_RETURN(cudaMemsetAsync(w.slip_dense.as<double>() + (size_t)s * 2 * gc.nf, 0,
                                                   sizeof(double) * 2 * gc.nf, G->stream));
            }
        }
        if (taken == 0) return EQD_OK;
        CUDA_OR_RETURN(cudaMemcpyAsync(w.slip_node.p, hn.data(), sizeof(int) * cap, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(w.slip_comp.p, hc.data(), sizeof(int) * cap, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(w.status.p, hst.data(), cap, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(w.iters.p, hit.data(), sizeof(int) * cap, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(w.newmask.p, hnew.data(), cap, cudaMemcpyHostToDevice, G->stream));
        const int8_t *mask = w.newmask.as<int8_t>();
        const unsigned nb = (unsigned)(cap * G->nchunks);
        const long long cst = sp.colstride;
        zero_columns_kernel<double><<<nb, 256, 0, G->stream>>>(w.x64.as<double>(), gc.colstride, G->nchunks, mask);
        zero_columns_kernel<T><<<nb, 256, 0, G->stream>>>(w.v0.as<T>(), cst, G->nchunks, mask);
        zero_columns_kernel<T><<<nb, 256, 0, G->stream>>>(w.v1.as<T>(), cst, G->nchunks, mask);
        zero_columns_kernel<T><<<nb, 256, 0, G->stream>>>(w.v2.as<T>(), cst, G->nchunks, mask);
        if (mixed) zero_columns_kernel<float><<<nb, 256, 0, G->stream>>>(w.v3.as<float>(), cst, G->nchunks, mask);
        // Fused: the second direction buffer's plane padding must read as zero.
        if (fused) zero_columns_kernel<T><<<nb, 256, 0, G->stream>>>(w.v4.as<T>(), cst, G->nchunks, mask);
        launches += (mixed ? 5 : 4) + (fused ? 1 : 0);
        const unsigned sb = (unsigned)((cap + 3) / 4);
        if (!generic) {
            // r0 = b = H P (D+SAT) chi  (x = 0), in the working precision.
            ColumnSet cs = colset();
            cs.flag = mask;
            cs.dinv = sp.precond ? G->dinv64.as<double>() : nullptr;
            CUDA_OR_RETURN((launch_march<double, T, MODE_RHS>(G, w.x64.as<double>(), xm ? w.v2.as<T>() : w.v0.as<T>(), cs,
                                                               w.res_part.as<double>(), cap)));
            SolveParams sp2 = sp;
            sp2.ntiles = nparts(G->m64);
            if (xm) launch_xresidual(G, w.v0.as<float>(), w.v1.as<float>(), w.v2.as<float>(), w.status.as<int8_t>(), mask, cap, G->stream);
            cg_true_residual_kernel<<<sb, 128, 0, G->stream>>>(st, sp2, w.res_part.as<double>(), cap, mixed, mask);
            launches += 2 + (xm ? 1 : 0);
        } else {
            // r0 = b given explicitly (reference layout, FP64).
            int j = 0;
            for (int s = 0; s < cap && j < taken; ++s) {
                if (!hnew[s]) continue;
                const ColWork &c = work[j++];
                double *hb = w.hbuf.as<double>() + (size_t)s * ntot;
                CUDA_OR_RETURN(cudaMemcpyAsync(hb, c.rhs, sizeof(double) * ntot, cudaMemcpyHostToDevice, G->stream));
                const int tb = 256;
                ref_to_dev_kernel<double, T><<<(unsigned)((ntot + tb - 1) / tb), tb, 0, G->stream>>>(
                    hb, w.v0.as<T>() + (size_t)s * gc.colstride, gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, 1);
                ++launches;
            }
            column_sumsq_kernel<T><<<nb, 256, 0, G->stream>>>(w.v0.as<T>(), cst, G->nchunks, mask,
                                                               w.res_part.as<double>(),
                                                               sp.precond ? G->dinv64.as<double>() : nullptr);
            SolveParams sp2 = sp;
            sp2.ntiles = G->nchunks;
            cg_true_residual_kernel<<<sb, 128, 0, G->stream>>>(st, sp2, w.res_part.as<double>(), cap, 0, mask);
            launches += 2;
        }
        if (resident || xm) {  // the kernel forms the first direction, p = r + 0 p, or it is formed with r
            CUDA_OR_RETURN(cudaGetLastError());
            return EQD_OK;
        }
        const T *dinvT = !sp.precond ? nullptr
                                     : (const T *)(sizeof(T) == 4 ? (const void *)G->dinv32.p : (const void *)G->dinv64.p);
        cg_pupdate_kernel<T><<<nb, 256, 0, G->stream>>>(w.v1.as<T>(), w.v0.as<T>(), st, sp, mask, dinvT, cap);
        ++launches;
        CUDA_OR_RETURN(cudaGetLastError());
        return EQD_OK;
    }

    // Run kIter iterations (when a column is running) and queue the status
    // read-back; collect() then lists the finished slots. Split in two so that
    // a caller driving several grids can have all of them running at once.
    int launch() {
        Workspace &w = *W;
        int running = 0;
        for (int s = 0; s < cap; ++s) running += tag[s] >= 0 && hst[s] == COL_ACTIVE;
        if (running > 0) {
            CUDA_OR_RETURN(cudaGraphLaunch(w.graph, G->stream));
            if (resident) launches += (int64_t)rounds * (mixed ? 4 : 1);
            else launches += (int64_t)kIter * ((mixed ? 7 : 4) - (fused ? 1 : 0)) * (w.graph_split ? 2 : 1);
        }
        CUDA_OR_RETURN(cudaMemcpyAsync(hst.data(), w.status.p, cap, cudaMemcpyDeviceToHost, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(hit.data(), w.iters.p, sizeof(int) * cap, cudaMemcpyDeviceToHost, G->stream));
        return EQD_OK;
    }

    int advance(std::vector<ColDone> &done) {
        int rc = launch();
        return rc ? rc : collect(done);
    }

    // Wait for the queued iterations; list the occupied slots whose status is
    // final.
    int collect(std::vector<ColDone> &done) {
        done.clear();
        Workspace &w = *W;
        CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
        int rc = check_device_error(G);
        if (rc) return rc;
        bool forced = false;
        for (int s = 0; s < cap; ++s) {
            if (tag[s] < 0) continue;
            if (hst[s] == COL_ACTIVE && hit[s] <= seen[s])
                return fail(EQD_ERR_CUDA, "a launch of CG iterations left an active column where it was");
            seen[s] = hit[s];
            if (hst[s] == COL_ACTIVE && hit[s] > itmax + 2 * std::max(kIter, resident ? kmax * rounds : 0)) {  // defensive: the kernels stop at itmax
                hst[s] = COL_MAXITER;
                forced = true;
            }
            if (hst[s] != COL_ACTIVE) done.push_back(ColDone{tag[s], s, hit[s], hst[s]});
        }
        if (forced)
            CUDA_OR_RETURN(cudaMemcpyAsync(w.status.p, hst.data(), cap, cudaMemcpyHostToDevice, G->stream));
        return EQD_OK;
    }

    // K columns of finished slots: into K (device) at column dst (the tag when
    // `to_tag`, else the position in `done`), leading dimension kld.
    int extract(const std::vector<ColDone> &done, double *K, long long kld, bool to_tag) {
        if (done.empty()) return EQD_OK;
        const GridConst &gc = G->gc;
        Workspace &w = *W;
        const int n = (int)done.size();
        for (int j = 0; j < n; ++j) {
            hslot[j] = done[j].slot;
            hdst[j] = to_tag ? (int)done[j].tag : j;
        }
        CUDA_OR_RETURN(cudaMemcpyAsync(w.slot_list.p, hslot.data(), sizeof(int) * n, cudaMemcpyHostToDevice, G->stream));
        CUDA_OR_RETURN(cudaMemcpyAsync(w.dst_list.p, hdst.data(), sizeof(int) * n, cudaMemcpyHostToDevice, G->stream));
        ExtractGeom eg{gc.n1, gc.n2, gc.n3, gc.PS, gc.nf, gc.i2f0, gc.n2f, gc.i3f0, gc.n3f, gc.colstride, gc.mu};
        const long long nthr = (long long)n * gc.nf;
        extract_traction_kernel<<<(unsigned)((nthr + 127) / 128), 128, 0, G->stream>>>(
            G->c64, eg, w.x64.as<double>(), colset(), K, kld, n, w.slot_list.as<int>(), w.dst_list.as<int>());
        ++launches;
        CUDA_OR_RETURN(cudaGetLastError());
        return EQD_OK;
    }

    // Explicit-RHS solve: the solution of a finished slot in reference layout.
    int solution(int slot, double *host_u) {
        const GridConst &gc = G->gc;
        const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
        Workspace &w = *W;
        double *hb = w.hbuf.as<double>() + (size_t)slot * ntot;
        const int tb = 256;
        dev_to_ref_kernel<double, double><<<(unsigned)((ntot + tb - 1) / tb), tb, 0, G->stream>>>(
            w.x64.as<double>() + (size_t)slot * gc.colstride, hb, gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, 1);
        ++launches;
        CUDA_OR_RETURN(cudaMemcpyAsync(host_u, hb, sizeof(double) * ntot, cudaMemcpyDeviceToHost, G->stream));
        return EQD_OK;
    }

    // Free the slots of finished columns.
    int release(const std::vector<ColDone> &done) {
        if (done.empty()) return EQD_OK;
        for (const ColDone &d : done) {
            tag[d.slot] = -1;
            hn[d.slot] = -1;
            hst[d.slot] = COL_IDLE;
            --held;
        }
        CUDA_OR_RETURN(cudaMemcpyAsync(W->status.p, hst.data(), cap, cudaMemcpyHostToDevice, G->stream));
        return EQD_OK;
    }
};

// Launch-variant tuner: time 20 CG iterations (two graph launches) of a
// batch of `ncols` unit-slip columns with each FP32 stencil variant and keep
// the fastest. The whole iteration is timed, not the stencil alone: a variant
// that packs more stencil CTAs per SM can leave less room for the other
// half's vector kernels (measured at h = 50 m: the fastest stencil alone was
// not the fastest iteration).
static int tune_by_iterations(eqd_grid *G, const eqd_solve_opts &o, int ncols, bool with_resident) {
    const GridConst &gc = G->gc;
    ncols = std::max(1, std::min(ncols, 2 * gc.nf));
    std::vector<ColWork> work(ncols);
    for (int i = 0; i < ncols; ++i) {
        work[i].slip_node = (int)(((long long)i * 7919 + gc.nf / 2) % gc.nf);
        work[i].slip_comp = i & 1;
        work[i].tag = i;
    }
    eqd_solve_opts ot = o;
    ot.precision = EQD_PREC_MIXED;
    G->tuned = true;  // the slot engines below must not tune again
    double best = 1e30;
    int bestv = G->sel32;
    const int pin0 = G->pin;
    struct PinGuard {
        eqd_grid *G;
        int v;
        ~PinGuard() { G->pin = v; }
    } guard{G, pin0};
    if (with_resident) {
        int rc = ensure_resident<float>(G, G->res32);
        if (rc) return rc;
    }
    G->tune_ms[kResidentVariant] = 0.0;
    G->tune_ms[kXMarchVariant] = 0.0;
    for (int v = 0; v < (with_resident ? kAllVariants : kNumVariants); ++v) {
        // (A grid that a variant has no plan for streams; Jacobi streams x1-fastest.)
        if (v >= kNumVariants && ot.precond == EQD_PRECOND_JACOBI) continue;
        if (v == kResidentVariant && !G->res32.ok) continue;
        G->pin = v;
        if (v < kNumVariants) G->sel32 = v;
        SlotRun<float> R;
        Path path;
        int rc = choose_path<float>(G, ot, false, false, path);
        if (!rc) rc = R.setup(G, ot, ncols, false, false, path, true);
        if (rc) return rc;
        int taken = 0;
        rc = R.admit(work.data(), ncols, taken);
        if (!rc) rc = R.launch();  // first launch: warm-up
        if (rc) return rc;
        CUDA_OR_RETURN(cudaEventRecord(G->ev0, G->stream));
        rc = R.launch();
        if (!rc) rc = R.launch();
        if (rc) return rc;
        CUDA_OR_RETURN(cudaEventRecord(G->ev1, G->stream));
        CUDA_OR_RETURN(cudaEventSynchronize(G->ev1));
        float ms = 0.f;
        CUDA_OR_RETURN(cudaEventElapsedTime(&ms, G->ev0, G->ev1));
        G->tune_ms[v] = ms / (2.0 * SlotRun<float>::kIter);
        if (G->tune_ms[v] < best) {
            best = G->tune_ms[v];
            bestv = v;
        }
    }
    // The streamed variant for what does not run resident, then the choice.
    G->sel32 = (int)(std::min_element(G->tune_ms, G->tune_ms + kNumVariants) - G->tune_ms);
    if (with_resident) guard.v = bestv;
    return check_device_error(G);
}

// Whether P b = b exactly: zero at the outer boundary, the same on both sides
// of every fault node. CG then stays in the range of P, which is all that the
// resident kernel holds; b = H P (...) always is, and what is not takes the
// streamed path, whose operator projects its input.
static bool rhs_in_range(const GridConst &gc, const double *b) {
    const int n1 = gc.n1, n2 = gc.n2, n3 = gc.n3;
    const long long pl = (long long)n1 * n2, comp = pl * n3, side = 3 * comp;
    for (int c = 0; c < 3; ++c)
        for (int i3 = 0; i3 < n3; ++i3)
            for (int i2 = 0; i2 < n2; ++i2) {
                const double *m = b + c * comp + i3 * pl + (long long)i2 * n1, *p = m + side;
                if (!(m[0] == 0.0 && p[n1 - 1] == 0.0 && m[n1 - 1] == p[0])) return false;
                if (i3 > 0 && i3 < n3 - 1 && i2 > 0 && i2 < n2 - 1) continue;
                for (int i = 0; i < n1; ++i)
                    if (!(m[i] == 0.0 && p[i] == 0.0)) return false;
            }
    return true;
}

// The explicit right-hand sides that run on chip: those in the range of P, each
// for itself, on a grid with a plan. Where the plan is a team that only a few
// columns are better off with, all of them while they are at most four a team.
// That number is the call's, whatever width the memory allows, so a right-hand
// side's bits depend on the call only where it is crossed.
template <typename T>
static int explicit_on_chip(eqd_grid *G, const eqd_solve_opts &o, const BatchSpec &B, std::vector<char> &on) {
    on.assign(B.ncols, 0);
    if (!allows_resident<T>(G, o)) return EQD_OK;
    ResEngine &E = sizeof(T) == 4 ? G->res32 : G->res64;
    int rc = ensure_resident<T>(G, E);
    if (rc || !E.ok) return rc;
    const size_t ntot = (size_t)6 * G->gc.n1 * G->gc.n2 * G->gc.n3;
    int n = 0;
    for (int i = 0; i < B.ncols; ++i) {
        n += on[i] = rhs_in_range(G->gc, B.rhs + i * ntot);
        if (E.few && n > 4 * E.teams) {  // (the rest need not be looked at)
            on.assign(B.ncols, 0);
            break;
        }
    }
    return EQD_OK;
}

// Batched solve through the slot engine: columns enter as slots free up; K
// columns go to the caller's device or host buffer as each column finishes.
// `work`: the call's columns that run alike; adds to *stats and to unconv.
template <typename T>
static int run_columns(eqd_grid *G, const eqd_solve_opts &o, const BatchSpec &B, const std::vector<ColWork> &work,
                       bool on_chip, eqd_stats *stats, int64_t &unconv_all) {
    const GridConst &gc = G->gc;
    const int generic = B.rhs != nullptr, ncols = (int)work.size();
    const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
    int chunk = 0;
    Path path;
    int rc = resolve_chunk<T>(G, o, ncols, generic, on_chip, path, chunk);
    if (rc) return rc;
    SlotRun<T> R;
    rc = R.setup(G, o, chunk, generic, B.slip_dense != nullptr, path);
    if (rc) return rc;
    int64_t tot_it = 0, max_it = 0, unconv = 0;
    PinnedArr<double> &kstage = R.W->kstage;
    if (!generic && B.kcols && !B.kdev && kstage.n < 2 * gc.nf * chunk)
        CUDA_OR_RETURN(kstage.assign(2 * gc.nf * chunk, 0.0));
    // Host K output: finished columns are staged in pinned memory, and the
    // host copies them to the caller's K after the next graph launch, while
    // the GPU runs those iterations.
    const bool host_k = !generic && B.kcols && !B.kdev;
    cudaEvent_t kready = nullptr;  // the staged columns have landed
    if (host_k) CUDA_OR_RETURN(cudaEventCreateWithFlags(&kready, cudaEventDisableTiming));
    struct EventGuard {
        cudaEvent_t e;
        ~EventGuard() {
            if (e) cudaEventDestroy(e);
        }
    } kready_guard{kready};
    std::vector<ColDone> staged;
    auto copy_staged = [&]() -> int {
        if (staged.empty()) return EQD_OK;
        CUDA_OR_RETURN(cudaEventSynchronize(kready));
        for (size_t j = 0; j < staged.size(); ++j)
            std::memcpy(B.kcols + (size_t)staged[j].tag * 2 * gc.nf, kstage.data() + j * 2 * gc.nf,
                        sizeof(double) * 2 * gc.nf);
        staged.clear();
        return EQD_OK;
    };
    CUDA_OR_RETURN(cudaEventRecord(G->ev0, G->stream));
    int next = 0, finished = 0;
    std::vector<ColDone> done;
    while (finished < ncols) {
        // Explicit-RHS solves refill only an empty engine (their staging
        // buffer holds one wave of right-hand sides).
        if (next < ncols && R.free_slots() > 0 && (!generic || R.held == 0)) {
            int taken = 0;
            rc = R.admit(work.data() + next, ncols - next, taken);
            if (rc) return rc;
            next += taken;
        }
        rc = R.launch();
        if (!rc) rc = copy_staged();
        if (!rc) rc = R.collect(done);
        if (rc) return rc;
        if (done.empty()) continue;
        if (!generic) {
            if (B.kdev) {
                rc = R.extract(done, B.kdev, 2LL * gc.nf, true);
            } else {
                rc = R.extract(done, R.W->kout.template as<double>(), 2LL * gc.nf, false);
                if (!rc && B.kcols) {
                    CUDA_OR_RETURN(cudaMemcpyAsync(kstage.data(), R.W->kout.p, sizeof(double) * 2 * gc.nf * done.size(),
                                                   cudaMemcpyDeviceToHost, G->stream));
                    CUDA_OR_RETURN(cudaEventRecord(kready, G->stream));
                    staged = done;
                }
            }
            if (rc) return rc;
        } else if (B.u_out) {
            for (const ColDone &d : done) {
                rc = R.solution(d.slot, B.u_out + (size_t)d.tag * ntot);
                if (rc) return rc;
            }
            CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
        }
        for (size_t j = 0; j < done.size(); ++j) {
            const ColDone &d = done[j];
            tot_it += d.iters;
            max_it = std::max<int64_t>(max_it, d.iters);
            if (d.status != COL_CONVERGED) ++unconv;
            if (B.iters) B.iters[d.tag] = d.iters;
            if (B.status) B.status[d.tag] = d.status;
        }
        finished += (int)done.size();
        rc = R.release(done);
        if (rc) return rc;
    }
    rc = copy_staged();
    if (rc) return rc;
    CUDA_OR_RETURN(cudaEventRecord(G->ev1, G->stream));
    CUDA_OR_RETURN(cudaEventSynchronize(G->ev1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, G->ev0, G->ev1);
    if (stats) {
        stats->solves += ncols;
        stats->iterations += tot_it;
        stats->max_iterations = std::max<int64_t>(stats->max_iterations, max_it);
        stats->unconverged += unconv;
        stats->kernel_launches += R.launches;
        stats->device_seconds += ms * 1e-3;
        stats->precision = o.precision;
        stats->precond = o.precond;
    }
    unconv_all += unconv;
    return EQD_OK;
}

template <typename T>
static int run_batch(eqd_grid *G, const eqd_solve_opts &o, const BatchSpec &B, eqd_stats *stats) {
    const GridConst &gc = G->gc;
    const long long ntot = 6LL * gc.n1 * gc.n2 * gc.n3;
    std::vector<char> on(B.ncols, 0);
    if (B.rhs) {
        int rc = explicit_on_chip<T>(G, o, B, on);
        if (rc) return rc;
    }
    std::vector<ColWork> work[2];  // explicit right-hand sides: streamed, on chip
    for (int i = 0; i < B.ncols; ++i) {
        ColWork c;
        c.tag = i;
        c.slip_node = B.slip_node ? B.slip_node[i] : -1;
        c.slip_comp = B.slip_comp ? B.slip_comp[i] : 0;
        c.slip_dense = B.slip_dense ? B.slip_dense + (size_t)i * 2 * gc.nf : nullptr;
        c.rhs = B.rhs ? B.rhs + (size_t)i * ntot : nullptr;
        work[on[i] ? 1 : 0].push_back(c);
    }
    int64_t unconv = 0;
    for (int k = 0; k < 2; ++k) {
        if (work[k].empty() && (k > 0 || !work[1].empty())) continue;
        int rc = run_columns<T>(G, o, B, work[k], k > 0, stats, unconv);
        if (rc) return rc;
    }
    if ((o.flags & EQD_FLAG_STRICT) && unconv > 0)
        return fail(EQD_ERR_NOT_CONVERGED, std::to_string(unconv) + " column(s) did not converge");
    return EQD_OK;
}

static int run_batch_any(eqd_grid *G, const eqd_solve_opts *opts, const BatchSpec &B, eqd_stats *stats) {
    eqd_solve_opts o;
    if (opts) o = *opts;
    else eqd_default_opts(&o);
    if (!(o.rtol >= 0) || !(o.atol >= 0)) return fail(EQD_ERR_ARG, "rtol/atol must be non-negative");
    if (o.precond != EQD_PRECOND_NONE && o.precond != EQD_PRECOND_JACOBI)
        return fail(EQD_ERR_ARG, "precond must be :none or :jacobi");
    if (o.precision != EQD_PREC_FP64 && o.precision != EQD_PREC_MIXED) return fail(EQD_ERR_ARG, "unknown precision");
    if (B.rhs && o.precision != EQD_PREC_FP64) return fail(EQD_ERR_UNSUPPORTED, "explicit-RHS solves run in FP64");
    if (o.variant < 0 || o.variant > kAllVariants)
        return fail(EQD_ERR_ARG, "variant must be 0 (the grid's) or 1.." + std::to_string(kAllVariants));
    const auto t0 = std::chrono::steady_clock::now();
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    // A per-call variant replaces the grid's selection for this call only.
    const int sel_before = G->sel32;
    const int pin_before = G->pin, pin64_before = G->pin64;
    const bool tuned_before = G->tuned;
    if (o.variant > 0) {
        G->pin = G->pin64 = o.variant - 1;
        if (G->pin < kNumVariants) {
            G->sel32 = G->pin;
            G->tuned = true;
        }
    }
    int rc = o.precision == EQD_PREC_MIXED ? run_batch<float>(G, o, B, stats) : run_batch<double>(G, o, B, stats);
    if (o.variant > 0) {
        G->pin = pin_before;
        G->pin64 = pin64_before;
        if (o.variant - 1 < kNumVariants) {
            G->sel32 = sel_before;
            G->tuned = tuned_before;
        }
    }
    if (stats)
        stats->seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return rc;
}

extern "C" int eqd_stiffness_columns(eqd_grid *G, const int32_t *cols, int32_t ncols, const eqd_solve_opts *opts,
                                     double *out, int32_t *iters, int8_t *status, eqd_stats *stats) {
    if (!G || (!cols && ncols > 0) || (!out && ncols > 0)) return fail(EQD_ERR_ARG, "null argument");
    if (ncols < 0) return fail(EQD_ERR_ARG, "ncols must be >= 0");
    if (ncols == 0) return EQD_OK;
    const int nf = G->gc.nf;
    std::vector<int> node(ncols), comp(ncols);
    for (int i = 0; i < ncols; ++i) {
        if (cols[i] < 0 || cols[i] >= 2 * nf) return fail(EQD_ERR_ARG, "column index out of range");
        node[i] = cols[i] < nf ? cols[i] : cols[i] - nf;
        comp[i] = cols[i] < nf ? 0 : 1;
    }
    BatchSpec B{};
    B.ncols = ncols;
    B.slip_node = node.data();
    B.slip_comp = comp.data();
    B.kcols = out;
    B.iters = iters;
    B.status = status;
    return run_batch_any(G, opts, B, stats);
}

extern "C" int eqd_stiffness_columns_device(eqd_grid *G, const int32_t *cols, int32_t ncols,
                                            const eqd_solve_opts *opts, double *out_device, int32_t *iters,
                                            int8_t *status, eqd_stats *stats) {
    if (!G || (!cols && ncols > 0) || (!out_device && ncols > 0)) return fail(EQD_ERR_ARG, "null argument");
    if (ncols < 0) return fail(EQD_ERR_ARG, "ncols must be >= 0");
    if (ncols == 0) return EQD_OK;
    cudaPointerAttributes pa{};
    if (cudaPointerGetAttributes(&pa, out_device) != cudaSuccess || pa.type != cudaMemoryTypeDevice ||
        pa.device != G->desc.device) {
        cudaGetLastError();
        return fail(EQD_ERR_ARG, "out_device is not device memory of the grid's device");
    }
    const int nf = G->gc.nf;
    std::vector<int> node(ncols), comp(ncols);
    for (int i = 0; i < ncols; ++i) {
        if (cols[i] < 0 || cols[i] >= 2 * nf) return fail(EQD_ERR_ARG, "column index out of range");
        node[i] = cols[i] < nf ? cols[i] : cols[i] - nf;
        comp[i] = cols[i] < nf ? 0 : 1;
    }
    BatchSpec B{};
    B.ncols = ncols;
    B.slip_node = node.data();
    B.slip_comp = comp.data();
    B.kdev = out_device;
    B.iters = iters;
    B.status = status;
    return run_batch_any(G, opts, B, stats);
}

extern "C" int eqd_stiffness_exact(eqd_grid *G, const eqd_solve_opts *opts, double *K, eqd_stats *stats) {
    if (!G || !K) return fail(EQD_ERR_ARG, "null argument");
    const int n = 2 * G->gc.nf;
    std::vector<int32_t> cols(n);
    for (int i = 0; i < n; ++i) cols[i] = i;
    return eqd_stiffness_columns(G, cols.data(), n, opts, K, nullptr, nullptr, stats);
}

extern "C" int eqd_shear_traction(eqd_grid *G, const double *s2, const double *s3, int32_t nslip, double *dtau2,
                                  double *dtau3, const eqd_solve_opts *opts, eqd_stats *stats) {
    if (!G || !s2 || !s3 || !dtau2 || !dtau3) return fail(EQD_ERR_ARG, "null argument");
    if (nslip < 1) return fail(EQD_ERR_ARG, "nslip must be >= 1");
    const int nf = G->gc.nf;
    std::vector<double> dense((size_t)nslip * 2 * nf);
    for (int c = 0; c < nslip; ++c)
        for (int k = 0; k < nf; ++k) {
            dense[((size_t)c * 2 + 0) * nf + k] = s2[(size_t)c * nf + k];
            dense[((size_t)c * 2 + 1) * nf + k] = s3[(size_t)c * nf + k];
        }
    std::vector<int> node(nslip, -1), comp(nslip, 0);
    std::vector<double> out((size_t)2 * nf * nslip);
    BatchSpec B{};
    B.ncols = nslip;
    B.slip_node = node.data();
    B.slip_comp = comp.data();
    B.slip_dense = dense.data();
    B.kcols = out.data();
    int rc = run_batch_any(G, opts, B, stats);
    if (rc) return rc;
    for (int c = 0; c < nslip; ++c)
        for (int k = 0; k < nf; ++k) {
            dtau2[(size_t)c * nf + k] = out[(size_t)c * 2 * nf + k];
            dtau3[(size_t)c * nf + k] = out[(size_t)c * 2 * nf + nf + k];
        }
    return EQD_OK;
}

extern "C" int eqd_cg_solve(eqd_grid *G, const double *rhs, double *u, int32_t ncols, const eqd_solve_opts *opts,
                            int32_t *iters, int8_t *status, eqd_stats *stats) {
    if (!G || !rhs || !u) return fail(EQD_ERR_ARG, "null argument");
    if (ncols < 1) return fail(EQD_ERR_ARG, "ncols must be >= 1");
    eqd_solve_opts o;
    if (opts) o = *opts;
    else eqd_default_opts(&o);
    o.precision = EQD_PREC_FP64;
    BatchSpec B{};
    B.ncols = ncols;
    B.rhs = rhs;
    B.u_out = u;
    B.iters = iters;
    B.status = status;
    return run_batch_any(G, &o, B, stats);
}

extern "C" int eqd_stiffness_toeplitz(eqd_grid *G, const eqd_solve_opts *opts, double *K, eqd_stats *stats) {
    if (!G || !K) return fail(EQD_ERR_ARG, "null argument");
    const GridConst &gc = G->gc;
    const int n2 = gc.n2f, n3 = gc.n3f, nf = gc.nf;
    // Sources in priority order: centre, then the corners (1-based (a, b)).
    const int ac = (n2 + 1) / 2, bc = (n3 + 1) / 2;
    const int sa[5] = {ac, 1, n2, 1, n2}, sb[5] = {bc, 1, 1, n3, n3};
    std::vector<int32_t> cols(10);
    for (int s = 0; s < 5; ++s) {
        const int node = (sb[s] - 1) * n2 + (sa[s] - 1);
        cols[2 * s] = node;
        cols[2 * s + 1] = nf + node;
    }
    std::vector<double> resp((size_t)10 * 2 * nf);
    int rc = eqd_stiffness_columns(G, cols.data(), 10, opts, resp.data(), nullptr, nullptr, stats);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    const size_t N = 2 * (size_t)nf;
    DevBuf dK, dsrc, da, db;
    CUDA_OR_RETURN(dK.ensure(sizeof(double) * N * N));
    CUDA_OR_RETURN(dsrc.ensure(sizeof(double) * resp.size()));
    CUDA_OR_RETURN(da.ensure(sizeof(int) * 5));
    CUDA_OR_RETURN(db.ensure(sizeof(int) * 5));
    CUDA_OR_RETURN(cudaMemcpyAsync(dsrc.p, resp.data(), sizeof(double) * resp.size(), cudaMemcpyHostToDevice, G->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(da.p, sa, sizeof(sa), cudaMemcpyHostToDevice, G->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(db.p, sb, sizeof(sb), cudaMemcpyHostToDevice, G->stream));
    const long long ne = (long long)nf * nf;
    toeplitz_expand_kernel<<<(unsigned)((ne + 255) / 256), 256, 0, G->stream>>>(dsrc.as<double>(), da.as<int>(),
                                                                              db.as<int>(), 5, n2, n3, dK.as<double>());
    CUDA_OR_RETURN(cudaGetLastError());
    CUDA_OR_RETURN(cudaMemcpyAsync(K, dK.p, sizeof(double) * N * N, cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    return EQD_OK;
}

// Whether streamed mixed-precision solves of this grid apply the x1 march.
static int streams_xmarch(eqd_grid *G, bool &xm) {
    xm = false;
    if (G->pin >= 0 && G->pin != kResidentVariant && G->pin != kXMarchVariant) return EQD_OK;
    int rc = ensure_resident<float>(G, G->res32);
    if (rc || (G->res32.ok && G->pin != kXMarchVariant)) return rc;
    rc = ensure_xmarch(G);
    xm = !rc && G->xm.ok;
    return rc;
}

template <typename T>
static int profile_apply_impl(eqd_grid *G, int ncols, int warmup, int reps, double *ms, double *bytes) {
    const GridConst &gc = G->gc;
    DevBuf x, y, part;
    bool xm = false;
    if (sizeof(T) == 4) {
        int rc = streams_xmarch(G, xm);
        if (rc) return rc;
    }
    const long long n = (xm ? G->xm.g.colstride : gc.colstride) * (long long)ncols;
    CUDA_OR_RETURN(x.ensure(sizeof(T) * n));
    CUDA_OR_RETURN(y.ensure(sizeof(T) * n));
    if (sizeof(T) == 4 && !xm && !G->tuned) {
        eqd_solve_opts o;
        eqd_default_opts(&o);
        int rc = tune_by_iterations(G, o, std::min(ncols, 1024));
        if (rc) return rc;
    }
    int nt = nparts(G->m64);
    for (int v = 0; v < kNumVariants; ++v) nt = std::max(nt, nparts(G->v32[v]));
    if (xm) nt = std::max(nt, G->xm.g.nt2 * G->xm.g.nt3);
    CUDA_OR_RETURN(part.ensure(sizeof(double) * 2 * ncols * nt));
    CUtensorMap map{};
    if (xm) {
        int rc = make_plane_map(G->xm.g, x.as<float>(), ncols, map);
        if (rc) return rc;
    }
    fill_random_kernel<T><<<1184, 256, 0, G->stream>>>(x.as<T>(), n, 12345ull);
    CUDA_OR_RETURN(cudaGetLastError());
    ColumnSet cs{};
    auto apply = [&]() -> cudaError_t {
        if (xm) return launch_xmarch(G, map, y.as<float>(), nullptr, part.as<double>(), 0, ncols, G->stream);
        return launch_march<T, T, MODE_A>(G, x.as<T>(), y.as<T>(), cs, part.as<double>(), ncols);
    };
    for (int i = 0; i < warmup; ++i) CUDA_OR_RETURN(apply());
    CUDA_OR_RETURN(cudaEventRecord(G->ev0, G->stream));
    for (int i = 0; i < reps; ++i) CUDA_OR_RETURN(apply());
    CUDA_OR_RETURN(cudaEventRecord(G->ev1, G->stream));
    CUDA_OR_RETURN(cudaEventSynchronize(G->ev1));
    float t = 0.f;
    CUDA_OR_RETURN(cudaEventElapsedTime(&t, G->ev0, G->ev1));
    if (ms) *ms = (double)t / std::max(reps, 1);
    if (bytes) *bytes = 2.0 * 6.0 * gc.n1 * gc.n2 * gc.n3 * sizeof(T) * ncols;
    return check_device_error(G);
}

extern "C" int eqd_profile_apply(eqd_grid *G, int32_t ncols, int32_t precision, int32_t warmup, int32_t reps,
                                 double *ms_per_launch, double *bytes_per_launch) {
    if (!G || ncols < 1 || reps < 1 || warmup < 0) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    if (precision == EQD_PREC_MIXED) return profile_apply_impl<float>(G, ncols, warmup, reps, ms_per_launch, bytes_per_launch);
    if (precision == EQD_PREC_FP64) return profile_apply_impl<double>(G, ncols, warmup, reps, ms_per_launch, bytes_per_launch);
    return fail(EQD_ERR_ARG, "unknown precision");
}

extern "C" int eqd_autotune(eqd_grid *G, int32_t ncols, int32_t *selected, double *ms_per_variant,
                            int32_t *tile_rows, int32_t *threads, int32_t *nvariants) {
    if (!G || ncols < 0) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    if (ncols > 0) {
        eqd_solve_opts o;
        eqd_default_opts(&o);
        int rc = tune_by_iterations(G, o, ncols, true);
        if (rc) return rc;
    }
    // (Nothing pinned: what the grid's solves have run with.)
    if (selected) *selected = G->pin >= 0 ? G->pin : G->res32.ok ? kResidentVariant : G->xm.ok ? kXMarchVariant : G->sel32;
    if (nvariants) *nvariants = kAllVariants;
    for (int v = kNumVariants; v < kAllVariants; ++v) {
        if (ms_per_variant) ms_per_variant[v] = G->tune_ms[v];
        if (tile_rows) tile_rows[v] = v == kXMarchVariant ? kXT2 : 0;
    }
    if (threads) threads[kXMarchVariant] = kXThreads;
    if (threads) threads[kResidentVariant] = G->res32.ok ? 64 * G->res32.d.nch0max : 0;
    for (int v = 0; v < kNumVariants; ++v) {
        if (ms_per_variant) ms_per_variant[v] = G->tune_ms[v];
        if (tile_rows) tile_rows[v] = G->v32[v].g.t2max;
        if (threads) threads[v] = G->v32[v].threads;
    }
    return EQD_OK;
}

// Chunk-width tuner: the cost of one column-iteration of the mixed-precision
// CG at each batch width (unit-slip columns, two graph launches = 20
// iterations after one untimed launch), and the cheapest width, which later
// calls with opts.chunk = 0 use (capped by the HBM budget).
extern "C" int eqd_tune_chunk(eqd_grid *G, const int32_t *widths, int32_t nwidths, double *ms_per_column_iteration,
                              int32_t *best) {
    if (!G || !widths || nwidths < 1) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    const GridConst &gc = G->gc;
    eqd_solve_opts o;
    eqd_default_opts(&o);
    int cap = 0;
    Path path;
    int rc = resolve_chunk<float>(G, o, 2 * gc.nf, false, false, path, cap);
    if (rc) return rc;
    double bestms = 1e300;
    int bestw = 0;
    for (int k = 0; k < nwidths; ++k) {
        const int w = widths[k];
        if (w < 1 || w > 2 * gc.nf || w > cap) {
            if (ms_per_column_iteration) ms_per_column_iteration[k] = -1.0;  // not measured: out of range
            continue;
        }
        std::vector<ColWork> work(w);
        for (int i = 0; i < w; ++i) {
            work[i].slip_node = (int)(((long long)i * 7919 + gc.nf / 2) % gc.nf);
            work[i].slip_comp = i & 1;
            work[i].tag = i;
        }
        SlotRun<float> R;
        rc = R.setup(G, o, w, false, false, path, true);
        if (rc) return rc;
        int taken = 0;
        rc = R.admit(work.data(), w, taken);
        if (!rc) rc = R.launch();
        if (rc) return rc;
        CUDA_OR_RETURN(cudaEventRecord(G->ev0, G->stream));
        rc = R.launch();
        if (!rc) rc = R.launch();
        if (rc) return rc;
        CUDA_OR_RETURN(cudaEventRecord(G->ev1, G->stream));
        CUDA_OR_RETURN(cudaEventSynchronize(G->ev1));
        float ms = 0.f;
        CUDA_OR_RETURN(cudaEventElapsedTime(&ms, G->ev0, G->ev1));
        const double per = ms / (2.0 * SlotRun<float>::kIter * w);
        if (ms_per_column_iteration) ms_per_column_iteration[k] = per;
        if (per < bestms) {
            bestms = per;
            bestw = w;
        }
    }
    if (bestw == 0) return fail(EQD_ERR_ARG, "no width within 1 .. min(2 nf, the budget's columns)");
    G->chunk_tuned = bestw;
    if (best) *best = bestw;
    return check_device_error(G);
}

extern "C" int eqd_set_variant(eqd_grid *G, int32_t variant) {
    if (!G || variant < 0 || variant >= kAllVariants) return fail(EQD_ERR_ARG, "invalid variant");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    G->pin = G->pin64 = variant;
    if (variant < kNumVariants) {
        G->sel32 = variant;
        G->tuned = true;
    }
    return EQD_OK;
}

extern "C" int eqd_test_inject_failure(eqd_grid *G, int32_t where) {
    if (!G || (where != EQD_FAIL_CG_LAUNCH && where != EQD_FAIL_PLAN)) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    (where == EQD_FAIL_CG_LAUNCH ? G->test_fail_launch : G->test_fail_plan) = true;
    return EQD_OK;
}

extern "C" int eqd_test_inject_wait_timeout(eqd_grid *G, int32_t plane, uint32_t poll_limit) {
    if (!G || plane < 0 || plane >= G->gc.n3 || poll_limit == 0) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    if (G->v32[G->sel32].ring_t2 <= 0)
        return fail(EQD_ERR_UNSUPPORTED, "the grid's FP32 apply variant is not a ring-march variant");
    G->test_drop_plane = plane;
    G->test_poll_limit = poll_limit;
    return EQD_OK;
}

// Sparse A (which = 0) or HP_DSAT (which = 1) in reference DOF order, CSR,
// by coloured probing with the FP64 operator kernels (probe_* kernels).
static constexpr int kProbeRowCap = 128;        // entries a row may hold before the drop (measured at most 96)
static constexpr double kProbeRelDrop = 1e-12;  // entries below this fraction of the row's largest are rounding

extern "C" int eqd_assemble(eqd_grid *G, int32_t which, int64_t capacity, int64_t *indptr, int32_t *indices,
                            double *values, int64_t *nnz) {
    if (!G || !nnz || (which != 0 && which != 1) || capacity < 0) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    const GridConst &gc = G->gc;
    ProbeGeom pg{};
    pg.n1 = gc.n1;
    pg.n2 = gc.n2;
    pg.n3 = gc.n3;
    pg.PS = gc.PS;
    pg.colstride = gc.colstride;
    pg.N = (long long)gc.n1 * gc.n2 * gc.n3;
    pg.R = 6;
    pg.P2 = gc.n2 <= 2 * pg.R + 1 ? gc.n2 : 2 * pg.R + 1;
    pg.P3 = gc.n3 <= 2 * pg.R + 1 ? gc.n3 : 2 * pg.R + 1;
    pg.ncolors = 6LL * gc.n1 * pg.P2 * pg.P3;
    const long long ntot = 6 * pg.N;
    if (ntot > INT32_MAX) return fail(EQD_ERR_UNSUPPORTED, "more DOFs than 32-bit column indices hold");
    // Probe chunk: at most 512 colours, within a quarter of free memory for x and y.
    size_t fr = 0, tot = 0;
    CUDA_OR_RETURN(cudaMemGetInfo(&fr, &tot));
    const size_t per = 2 * sizeof(double) * (size_t)gc.colstride;
    long long nc = std::min<long long>({512, pg.ncolors, (long long)(fr / 4 / per)});
    if (nc < 1) return fail(EQD_ERR_OOM, "no room for one probe");
    DevBuf x, y, sn, scomp, rcnt, rcol, rval, rmax, kept, dptr, dind, dval, ovf;
    CUDA_OR_RETURN(x.ensure(sizeof(double) * gc.colstride * nc));
    CUDA_OR_RETURN(y.ensure(sizeof(double) * gc.colstride * nc));
    CUDA_OR_RETURN(sn.ensure(sizeof(int) * nc));
    CUDA_OR_RETURN(scomp.ensure(sizeof(int) * nc));
    CUDA_OR_RETURN(rcnt.ensure(sizeof(int) * ntot));
    CUDA_OR_RETURN(rcol.ensure(sizeof(int) * ntot * kProbeRowCap));
    CUDA_OR_RETURN(rval.ensure(sizeof(double) * ntot * kProbeRowCap));
    CUDA_OR_RETURN(rmax.ensure(sizeof(double) * ntot));
    CUDA_OR_RETURN(kept.ensure(sizeof(long long) * ntot));
    CUDA_OR_RETURN(ovf.ensure(sizeof(unsigned)));
    cudaStream_t st = G->stream;
    CUDA_OR_RETURN(cudaMemsetAsync(rcnt.p, 0, sizeof(int) * ntot, st));
    CUDA_OR_RETURN(cudaMemsetAsync(rmax.p, 0, sizeof(double) * ntot, st));
    CUDA_OR_RETURN(cudaMemsetAsync(ovf.p, 0, sizeof(unsigned), st));
    {
        std::vector<int> neg(nc, -1);
        CUDA_OR_RETURN(cudaMemcpyAsync(sn.p, neg.data(), sizeof(int) * nc, cudaMemcpyHostToDevice, st));
        CUDA_OR_RETURN(cudaMemsetAsync(scomp.p, 0, sizeof(int) * nc, st));
        CUDA_OR_RETURN(cudaStreamSynchronize(st));
    }
    ColumnSet cs{};
    cs.slip_node = sn.as<int>();  // no slip: HP_DSAT x without the chi term
    cs.slip_comp = scomp.as<int>();
    const unsigned rb = (unsigned)((ntot + 255) / 256);
    for (long long c0 = 0; c0 < pg.ncolors; c0 += nc) {
        const int n = (int)std::min<long long>(nc, pg.ncolors - c0);
        CUDA_OR_RETURN(cudaMemsetAsync(x.p, 0, sizeof(double) * gc.colstride * n, st));
        probe_fill_kernel<<<1184, 256, 0, st>>>(pg, c0, n, x.as<double>());
        CUDA_OR_RETURN(cudaGetLastError());
        if (which == 0)
            CUDA_OR_RETURN((launch_march<double, double, MODE_AP>(G, x.as<double>(), y.as<double>(), cs, nullptr, n)));
        else
            CUDA_OR_RETURN((launch_march<double, double, MODE_RHS>(G, x.as<double>(), y.as<double>(), cs, nullptr, n)));
        probe_extract_kernel<<<rb, 256, 0, st>>>(pg, c0, n, y.as<double>(), kProbeRowCap, rcnt.as<int>(), rcol.as<int>(),
                                                 rval.as<double>(), rmax.as<double>(), ovf.as<unsigned>());
        CUDA_OR_RETURN(cudaGetLastError());
    }
    probe_compact_kernel<<<rb, 256, 0, st>>>(ntot, kProbeRowCap, rcnt.as<int>(), rcol.as<int>(), rval.as<double>(),
                                             rmax.as<double>(), kProbeRelDrop, 0, nullptr, nullptr, nullptr,
                                             kept.as<long long>());
    CUDA_OR_RETURN(cudaGetLastError());
    std::vector<long long> cnt(ntot);
    unsigned hovf = 0;
    CUDA_OR_RETURN(cudaMemcpyAsync(cnt.data(), kept.p, sizeof(long long) * ntot, cudaMemcpyDeviceToHost, st));
    CUDA_OR_RETURN(cudaMemcpyAsync(&hovf, ovf.p, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    CUDA_OR_RETURN(cudaStreamSynchronize(st));
    int rc = check_device_error(G);
    if (rc) return rc;
    if (hovf) return fail(EQD_ERR_UNSUPPORTED, "a row holds more than " + std::to_string(kProbeRowCap) + " entries");
    std::vector<long long> off(ntot + 1, 0);
    for (long long i = 0; i < ntot; ++i) off[i + 1] = off[i] + cnt[i];
    *nnz = off[ntot];
    if (!indptr && !indices && !values) return EQD_OK;  // size query
    if (!indptr || !indices || !values) return fail(EQD_ERR_ARG, "indptr, indices and values go together");
    if (capacity < off[ntot])
        return fail(EQD_ERR_ARG, "capacity " + std::to_string(capacity) + " below nnz " + std::to_string(off[ntot]));
    CUDA_OR_RETURN(dptr.ensure(sizeof(long long) * (ntot + 1)));
    CUDA_OR_RETURN(dind.ensure(sizeof(int) * std::max<long long>(off[ntot], 1)));
    CUDA_OR_RETURN(dval.ensure(sizeof(double) * std::max<long long>(off[ntot], 1)));
    CUDA_OR_RETURN(cudaMemcpyAsync(dptr.p, off.data(), sizeof(long long) * (ntot + 1), cudaMemcpyHostToDevice, st));
    probe_compact_kernel<<<rb, 256, 0, st>>>(ntot, kProbeRowCap, rcnt.as<int>(), rcol.as<int>(), rval.as<double>(),
                                             rmax.as<double>(), kProbeRelDrop, 1, dptr.as<long long>(), dind.as<int>(),
                                             dval.as<double>(), nullptr);
    CUDA_OR_RETURN(cudaGetLastError());
    CUDA_OR_RETURN(cudaMemcpyAsync(indices, dind.p, sizeof(int) * off[ntot], cudaMemcpyDeviceToHost, st));
    CUDA_OR_RETURN(cudaMemcpyAsync(values, dval.p, sizeof(double) * off[ntot], cudaMemcpyDeviceToHost, st));
    CUDA_OR_RETURN(cudaStreamSynchronize(st));
    for (long long i = 0; i <= ntot; ++i) indptr[i] = off[i];
    return EQD_OK;
}

extern "C" int eqd_diag(eqd_grid *G, double *d) {
    if (!G || !d) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to a server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    const GridConst &gc = G->gc;
    const long long n = 6LL * gc.n1 * gc.n2 * gc.n3;
    DevBuf dev, ref, neg;
    CUDA_OR_RETURN(dev.ensure(sizeof(double) * gc.colstride));
    CUDA_OR_RETURN(ref.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(neg.ensure(sizeof(unsigned)));
    CUDA_OR_RETURN(cudaMemsetAsync(neg.p, 0, sizeof(unsigned), G->stream));
    jacobi_diag_kernel<<<(unsigned)((n + 255) / 256), 256, 0, G->stream>>>(G->c64, gc.n1, gc.n2, gc.n3, gc.PS,
                                                                            dev.as<double>(), nullptr, nullptr,
                                                                            neg.as<unsigned>());
    dev_to_ref_kernel<double, double><<<(unsigned)((n + 255) / 256), 256, 0, G->stream>>>(
        dev.as<double>(), ref.as<double>(), gc.n1, gc.n2, gc.n3, gc.PS, gc.colstride, 1);
    CUDA_OR_RETURN(cudaGetLastError());
    CUDA_OR_RETURN(cudaMemcpyAsync(d, ref.p, sizeof(double) * n, cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Resident K and the time-loop GEMV
// ---------------------------------------------------------------------------
extern "C" int eqd_kmat_create(int32_t device, int32_t n, const double *K, eqd_kmat **out) {
    if (!out || !K || n < 1) return fail(EQD_ERR_ARG, "invalid argument");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
    if (device < 0 || device >= ndev) return fail(EQD_ERR_ARG, "device ordinal out of range");
    CUDA_OR_RETURN(cudaSetDevice(device));
    std::unique_ptr<eqd_kmat> M(new eqd_kmat());
    M->device = device;
    M->n = n;
    CUDA_OR_RETURN(M->K.ensure(sizeof(double) * (size_t)n * n));
    CUDA_OR_RETURN(cudaStreamCreateWithFlags(&M->stream, cudaStreamNonBlocking));
    int sms = 0, per_sm[3] = {0, 0, 0};
    CUDA_OR_RETURN(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    CUDA_OR_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[0], gemm_ks_dmma_kernel<true, 1, 32>, 256, 0));
    CUDA_OR_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[1], gemm_ks_dmma_kernel<true, 2, 32>, 256, 0));
    CUDA_OR_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[2], gemm_ks_dmma_kernel<true, 4, 16>, 256, 0));
    for (int k = 0; k < 3; ++k) M->ks_slots[k] = std::max(1, sms * per_sm[k]);
    CUDA_OR_RETURN(cudaMemcpyAsync(M->K.p, K, sizeof(double) * (size_t)n * n, cudaMemcpyHostToDevice, M->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(M->stream));
    *out = M.release();
    return EQD_OK;
}

// Row pairs of a cluster (gemv_kernel): the least of 32, 64 and 128 whose
// clusters run in one wave. 104 clusters of eight CTAs, six an SM, do on 148 SMs;
// 106 do not, although the CTAs alone would fit (n = 13,568: 279 us with one
// vector and 306 with two on 64 row pairs, 227 and 257 on 128; 6,784: 84 with two
// on 32, 70 on 64).
static int gemv_lx(long long n) { return n <= 104 * 64 ? 32 : n <= 104 * 128 ? 64 : 128; }

// y = K s, nothing of y in s.
static cudaError_t launch_gemv(cudaStream_t st, const double *K, const double *s, int n, int nvec, double *y) {
    const int nv = nvec >= 3 ? 4 : nvec, lx = gemv_lx(n);
    const long long tiles = (n + 2 * lx - 1) / (2 * lx), groups = ((long long)nvec + nv - 1) / nv;
    const unsigned gy = (unsigned)std::min<long long>(groups, 65535);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kGemvCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(tiles * kGemvCluster), gy, (unsigned)((groups + gy - 1) / gy));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const bool v2 = gemv_vec2_ok(K, n);
#define EQD_GEMV(NV)                                                                                            \
    if (nv == NV)                                                                                               \
        return cudaLaunchKernelEx(&cfg,                                                                         \
                                  lx == 32   ? (v2 ? gemv_kernel<true, NV, 32> : gemv_kernel<false, NV, 32>)    \
                                  : lx == 64 ? (v2 ? gemv_kernel<true, NV, 64> : gemv_kernel<false, NV, 64>)    \
                                             : (v2 ? gemv_kernel<true, NV, 128> : gemv_kernel<false, NV, 128>), \
                                  K, s, n, nvec, y)
    EQD_GEMV(1);
    EQD_GEMV(2);
    EQD_GEMV(4);
#undef EQD_GEMV
    return cudaErrorInvalidValue;
}

// The same for any s and y of `ne` values: a y that overlaps s is finished in `scratch` first.
static bool gemv_overlap(const double *s, const double *y, long long ne) { return s < y + ne && y < s + ne; }

static cudaError_t launch_gemv_any(cudaStream_t st, const double *K, const double *s, int n, int nvec, double *y,
                                   double *scratch) {
    const long long ne = (long long)n * nvec;
    if (!gemv_overlap(s, y, ne)) return launch_gemv(st, K, s, n, nvec, y);
    cudaError_t e = launch_gemv(st, K, s, n, nvec, scratch);
    return e != cudaSuccess ? e : cudaMemcpyAsync(y, scratch, sizeof(double) * ne, cudaMemcpyDeviceToDevice, st);
}

// Whether y = K s for nvec vectors runs as the GEMV (K read once per 4) or as
// the blocked K S on the FP64 tensor cores (once per 16 to 64). Measured, GEMV
// against blocked, us. 1 and 2 vectors: always (n = 4,356: 27, and 40 from 3 on
// blocked). More, while all groups of four are one wave, 71 clusters on 148 SMs:
// n = 4,544 3 and 4 vectors 32.5 against 41, and 53.5 against 41.5 at 4,600; n =
// 2,234 8 14.7 and 17.3, 1,400 12 10.6 and 12.9, 16 (88 clusters) 15.0 and 13.4.
// Beyond one wave where a wave is short: n = 1,000 48 19 and 23, 900 64 23 and 21;
// 1,156 24 15.8 and 15.8, 28 16.8 and 15.8; 1,300 16 14.7 and 13.8. Odd n has
// 8-byte loads: n = 3,001 4 22.7 and 24, 3,501 33 and 29; 801 32 15.5 and 17, 1,001
// 32 18.5 and 17.9, 1,157 16 (76 clusters) 17 and 13.8.
static bool gemv_better(long long n, int nvec) {
    const long long groups = (nvec + 3) / 4, reads = groups * n * n;
    const bool even = n % 2 == 0;
    if (nvec <= 2) return true;
    if (groups * ((n + 63) / 64) <= 71) return even || n <= 3200;
    if (n <= 1000) return reads <= (even ? 10000000 : 5500000);
    return even && n <= 1280 && reads <= 8200000;
}

// Column slices of the blocked K S: the count (1..16, slices of at least 128
// columns) with the least time in whole waves of resident CTAs,
// ceil(tiles * ns / slots) / ns; the smallest count on ties.
static int ks_slices(long long n, int nvec, int bn, int slots) {
    const long long tiles = ((n + kDmmaBM - 1) / kDmmaBM) * ((nvec + bn - 1) / bn);
    const int max_ns = (int)std::max<long long>(1, std::min<long long>(16, n / 128));
    int best = 1;
    double best_t = 1e300;
    for (int ns = 1; ns <= max_ns; ++ns) {
        const double tm = (double)((tiles * ns + slots - 1) / slots) / ns;
        if (tm < best_t * (1.0 - 1e-9)) {
            best_t = tm;
            best = ns;
        }
    }
    return best;
}

// y = K s for nvec device-resident vectors (s, y: n x nvec, column-major) on
// stream st; returns after the launches. Scratch: M->part.
static int kmat_apply(eqd_kmat *M, const double *s, double *y, int nvec, cudaStream_t st) {
    const int n = M->n;
    const long long ne = (long long)n * nvec;
    const double *K = M->K.as<double>();
    if (!gemv_better(n, nvec)) {
        // Vector tile: 16, 32 or 64 vectors per CTA, the narrowest that holds nvec.
        const int tk = nvec <= 16 ? 0 : nvec <= 32 ? 1 : 2, bn = 16 << tk;
        // The slice count depends only on n, nvec and the tile (the
        // occupancy of the 16-byte-load instance on either load path), so a
        // product is the same bits whatever the slips' alignment.
        const int ns = ks_slices(n, nvec, bn, M->ks_slots[tk]);
        CUDA_OR_RETURN(M->part.ensure(sizeof(double) * (size_t)ne * ns));
        const dim3 grid((unsigned)((n + kDmmaBM - 1) / kDmmaBM), (unsigned)ns, (unsigned)((nvec + bn - 1) / bn));
        const bool v2 = gemv_vec2_ok(K, n) && gemv_vec2_ok(s, n);
        double *pp = M->part.as<double>();
#define EQD_KS(V, NT) gemm_ks_dmma_kernel<V, NT, (NT < 4 ? 32 : 16)><<<grid, 256, 0, st>>>(K, s, n, ns, nvec, pp)
        if (tk == 0) { if (v2) EQD_KS(true, 1); else EQD_KS(false, 1); }
        else if (tk == 1) { if (v2) EQD_KS(true, 2); else EQD_KS(false, 2); }
        else { if (v2) EQD_KS(true, 4); else EQD_KS(false, 4); }
#undef EQD_KS
        gemv_reduce_kernel<<<(unsigned)((ne + 255) / 256), 256, 0, st>>>(M->part.as<double>(), n, ns, nvec, y);
    } else {
        // (Also where this call does not need it: the first call with an n * nvec allocates, and a
        // captured one after it, y over s or not, must not.)
        CUDA_OR_RETURN(M->part.ensure(sizeof(double) * (size_t)ne));
        CUDA_OR_RETURN(launch_gemv_any(st, K, s, n, nvec, y, M->part.as<double>()));
    }
    CUDA_OR_RETURN(cudaGetLastError());
    return EQD_OK;
}

extern "C" int eqd_kmat_gemv(eqd_kmat *M, const double *s, double *y, int32_t nvec) {
    if (!M || !s || !y || nvec < 1) return fail(EQD_ERR_ARG, "invalid argument");
    CUDA_OR_RETURN(cudaSetDevice(M->device));
    const size_t bytes = sizeof(double) * (size_t)M->n * nvec;
    CUDA_OR_RETURN(M->s.ensure(bytes));
    CUDA_OR_RETURN(M->y.ensure(bytes));
    CUDA_OR_RETURN(cudaMemcpyAsync(M->s.p, s, bytes, cudaMemcpyHostToDevice, M->stream));
    const int rc = kmat_apply(M, M->s.as<double>(), M->y.as<double>(), nvec, M->stream);
    if (rc) return rc;
    CUDA_OR_RETURN(cudaMemcpyAsync(y, M->y.p, bytes, cudaMemcpyDeviceToHost, M->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(M->stream));
    return EQD_OK;
}

extern "C" int eqd_kmat_gemv_device(eqd_kmat *M, const double *s_device, double *y_device, int32_t nvec,
                                    void *stream) {
    if (!M || !s_device || !y_device || nvec < 1) return fail(EQD_ERR_ARG, "invalid argument");
    if ((reinterpret_cast<uintptr_t>(s_device) & 7u) || (reinterpret_cast<uintptr_t>(y_device) & 7u))
        return fail(EQD_ERR_ARG, "s and y must be 8-byte aligned");
    CUDA_OR_RETURN(cudaSetDevice(M->device));
    return kmat_apply(M, s_device, y_device, nvec, static_cast<cudaStream_t>(stream));
}

extern "C" int eqd_kmat_destroy(eqd_kmat *M) {
    if (!M) return EQD_OK;
    cudaSetDevice(M->device);
    if (M->stream) {
        cudaStreamSynchronize(M->stream);
        cudaStreamDestroy(M->stream);
    }
    delete M;
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free GEMV.
//
// For callers that must not allocate device memory at all: a time loop that
// runs inside a CUDA graph or under a framework's own device allocator (a
// Julia CuArray pool, a PyTorch caching allocator), where a hidden cudaMalloc
// would break capture or fragment the caller's pool, and latency-critical
// loops that may not block on the allocator. The caller passes K, s and y as
// device pointers it already owns; the only scratch (the result, where y
// overlaps s) lives in this file-scope array, 4 MiB per device, held by every
// GPU that loads the library until exit. The first call on a device looks the
// array's device address up (with that device current); make that first call
// before any stream capture. Calls on a device with overlapping s and y share
// the array: where they overlap on the GPU they race, so serialise them (one
// stream, or events).
// ---------------------------------------------------------------------------
#define EQD_GEMV_STATIC_SCRATCH_DOUBLES (1 << 19)

static __device__ __align__(256) double g_gemv_static_scratch[EQD_GEMV_STATIC_SCRATCH_DOUBLES];

static std::mutex g_gemv_static_mtx;
static double *g_gemv_static_ptr[128] = {nullptr};

extern "C" int eqd_kmat_gemv_static(int32_t device, int32_t n, const double *K_device, const double *s_device,
                                    double *y_device, int32_t nvec, void *stream) {
    if (n < 1 || nvec < 1 || !K_device || !s_device || !y_device) return fail(EQD_ERR_ARG, "invalid argument");
    if ((long long)n * nvec > EQD_GEMV_STATIC_SCRATCH_DOUBLES)
        return fail(EQD_ERR_ARG, "eqd_kmat_gemv_static: n * nvec = " + std::to_string((long long)n * nvec) +
                                     " exceeds the static scratch of " +
                                     std::to_string(EQD_GEMV_STATIC_SCRATCH_DOUBLES) + " doubles");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
    if (device < 0 || device >= ndev || device >= 128) return fail(EQD_ERR_ARG, "device ordinal out of range");
    int prev = 0;
    CUDA_OR_RETURN(cudaGetDevice(&prev));
    if (prev != device) CUDA_OR_RETURN(cudaSetDevice(device));
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_gemv_static_mtx);
        if (!g_gemv_static_ptr[device]) {
            void *ptr = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&ptr, g_gemv_static_scratch);
            if (e != cudaSuccess) {
                if (prev != device) cudaSetDevice(prev);
                return fail(EQD_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
            }
            g_gemv_static_ptr[device] = static_cast<double *>(ptr);
        }
        scratch = g_gemv_static_ptr[device];
    }
    const cudaError_t e =
        launch_gemv_any(static_cast<cudaStream_t>(stream), K_device, s_device, n, nvec, y_device, scratch);
    if (prev != device) cudaSetDevice(prev);
    if (e != cudaSuccess) return fail(EQD_ERR_CUDA, std::string("eqd_kmat_gemv_static launch: ") + cudaGetErrorString(e));
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Server: continuous batching of stiffness-column requests across grids.
// Each attached grid has a slot engine and a worker thread of its own: it
// admits queued columns into free slots, runs the next graph of iterations
// on the grid's streams (grids overlap on the device), then collects
// finished columns and writes them to their requests' host buffers.
// ---------------------------------------------------------------------------
namespace {

struct SrvRequest {
    int64_t id = 0;
    double *k_out = nullptr;
    int ncols = 0, remaining = 0, unconverged = 0, max_it = 0;
    int64_t iterations = 0;
    int state = 0;  // 0 queued, 1 running, 2 done, 3 failed
    int err = EQD_OK;
    std::string msg;
    double t_submit = 0, t_start = -1, t_done = -1;
};

struct SrvGrid {
    eqd_grid *G = nullptr;
    int slots = 0;
    size_t bytes = 0;
    std::unique_ptr<SlotRun<float>> r32;
    std::unique_ptr<SlotRun<double>> r64;
    std::deque<ColWork> pending;  // guarded by the server mutex
    PinnedArr<double> kstage;     // finished K columns, compact
    std::vector<ColDone> done;
    std::thread worker;
    int held() const { return r32 ? r32->held : r64->held; }
    int free_slots() const { return r32 ? r32->free_slots() : r64->free_slots(); }
};

// Column tags carry the request id and the column's position in it.
constexpr int kTagBits = 24;

}  // namespace

struct eqd_server {
    eqd_solve_opts opts{};
    uint64_t budget = 0, used = 0;
    std::vector<std::unique_ptr<SrvGrid>> grids;
    std::map<int64_t, std::unique_ptr<SrvRequest>> reqs;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    bool stop = false;
    int64_t next_id = 1;
    int fatal = EQD_OK;
    std::string fatal_msg;
    std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
    double now() const { return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); }
};

static void server_fail_all(eqd_server *S, int code, const std::string &msg) {
    std::lock_guard<std::mutex> lk(S->mu);
    S->fatal = code;
    S->fatal_msg = msg;
    for (auto &kv : S->reqs) {
        SrvRequest &r = *kv.second;
        if (r.state < 2) {
            r.state = 3;
            r.err = code;
            r.msg = msg;
            r.t_done = S->now();
        }
    }
    for (auto &g : S->grids) g->pending.clear();
    S->cv_done.notify_all();
}

// Admission order of a grid's queued columns: the request with the fewest
// columns still queued goes first (a small request is not held behind the
// columns of a large one that arrived earlier), unless the oldest queued
// request has waited longer than kServeAgeLimit seconds, which then goes
// first (no request starves). A request's columns stay in submission order.
// Queued columns of one request are contiguous in `pending` (submit appends
// them under the server lock).
constexpr double kServeAgeLimit = 2.0;

static void take_columns(eqd_server *S, SrvGrid &g, int nfree, std::vector<ColWork> &take) {
    struct Run {
        size_t beg, len;
        double t_submit;
    };
    while ((int)take.size() < nfree && !g.pending.empty()) {
        std::vector<Run> runs;
        for (size_t i = 0; i < g.pending.size();) {
            const int64_t id = g.pending[i].tag >> kTagBits;
            size_t j = i + 1;
            while (j < g.pending.size() && (g.pending[j].tag >> kTagBits) == id) ++j;
            auto it = S->reqs.find(id);
            runs.push_back(Run{i, j - i, it != S->reqs.end() ? it->second->t_submit : 0.0});
            i = j;
        }
        size_t pick = 0;  // runs[0] is the oldest
        if (S->now() - runs[0].t_submit <= kServeAgeLimit)
            for (size_t k = 1; k < runs.size(); ++k)
                if (runs[k].len < runs[pick].len) pick = k;
        const Run r = runs[pick];
        const size_t n = std::min(r.len, (size_t)(nfree - (int)take.size()));
        for (size_t k = 0; k < n; ++k) take.push_back(g.pending[r.beg + k]);
        g.pending.erase(g.pending.begin() + (long)r.beg, g.pending.begin() + (long)(r.beg + n));
    }
}

// One pass of a grid's worker: admit queued columns into free slots, run
// the next graph of iterations, deliver the columns that finished.
static int grid_pass(eqd_server *S, SrvGrid &g) {
    eqd_grid *G = g.G;
    std::vector<ColWork> take;
    {
        std::lock_guard<std::mutex> lk(S->mu);
        take_columns(S, g, g.free_slots(), take);
        const double t = S->now();
        for (const ColWork &c : take) {
            auto it = S->reqs.find(c.tag >> kTagBits);
            if (it != S->reqs.end() && it->second->state == 0) {
                it->second->state = 1;
                it->second->t_start = t;
            }
        }
    }
    int rc = EQD_OK, taken = 0;
    if (!take.empty())
        rc = g.r32 ? g.r32->admit(take.data(), (int)take.size(), taken)
                   : g.r64->admit(take.data(), (int)take.size(), taken);
    if (rc) return rc;
    if (g.held() == 0) return EQD_OK;
    rc = g.r32 ? g.r32->advance(g.done) : g.r64->advance(g.done);
    if (rc) return rc;
    if (g.done.empty()) return EQD_OK;
    const int nf2 = 2 * G->gc.nf;
    rc = g.r32 ? g.r32->extract(g.done, G->ws.kout.as<double>(), nf2, false)
               : g.r64->extract(g.done, G->ws.kout.as<double>(), nf2, false);
    if (rc) return rc;
    CUDA_OR_RETURN(cudaMemcpyAsync(g.kstage.data(), G->ws.kout.p, sizeof(double) * nf2 * g.done.size(),
                                   cudaMemcpyDeviceToHost, G->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    {
        std::lock_guard<std::mutex> lk(S->mu);
        const double t = S->now();
        bool any_done = false;
        for (size_t j = 0; j < g.done.size(); ++j) {
            const ColDone &d = g.done[j];
            auto it = S->reqs.find(d.tag >> kTagBits);
            if (it == S->reqs.end()) continue;
            SrvRequest &r = *it->second;
            const long long pos = d.tag & ((1LL << kTagBits) - 1);
            std::memcpy(r.k_out + (size_t)pos * nf2, g.kstage.data() + j * nf2, sizeof(double) * nf2);
            r.iterations += d.iters;
            r.max_it = std::max(r.max_it, d.iters);
            if (d.status != COL_CONVERGED) ++r.unconverged;
            if (--r.remaining == 0) {
                r.state = 2;
                r.t_done = t;
                any_done = true;
            }
        }
        if (any_done) S->cv_done.notify_all();
    }
    return g.r32 ? g.r32->release(g.done) : g.r64->release(g.done);
}

// One worker thread per grid: a grid advances at its own pace (its graphs
// run on its own streams), so a request on a small grid is not held behind
// the long iterations of a large one.
static void grid_loop(eqd_server *S, SrvGrid *g) {
    if (cudaSetDevice(g->G->desc.device) != cudaSuccess) {
        server_fail_all(S, EQD_ERR_CUDA, "cudaSetDevice failed in a server worker");
        return;
    }
    for (;;) {
        {
            std::unique_lock<std::mutex> lk(S->mu);
            S->cv_work.wait(lk, [&] { return S->stop || S->fatal || !g->pending.empty() || g->held() > 0; });
            if (S->stop || S->fatal) return;
        }
        const int rc = grid_pass(S, *g);
        if (rc) {
            server_fail_all(S, rc, g_last_error);
            S->cv_work.notify_all();
            return;
        }
    }
}

extern "C" int eqd_server_create(const eqd_solve_opts *opts, uint64_t hbm_budget_bytes, eqd_server **out) {
    if (!out) return fail(EQD_ERR_ARG, "null argument");
    *out = nullptr;
    std::unique_ptr<eqd_server> S(new eqd_server());
    if (opts) S->opts = *opts;
    else eqd_default_opts(&S->opts);
    const eqd_solve_opts &o = S->opts;
    if (!(o.rtol >= 0) || !(o.atol >= 0)) return fail(EQD_ERR_ARG, "rtol/atol must be non-negative");
    if (o.precision != EQD_PREC_FP64 && o.precision != EQD_PREC_MIXED) return fail(EQD_ERR_ARG, "unknown precision");
    if (o.precond != EQD_PRECOND_NONE && o.precond != EQD_PRECOND_JACOBI)
        return fail(EQD_ERR_ARG, "precond must be :none or :jacobi");
    S->budget = hbm_budget_bytes;
    if (S->budget == 0) {
        size_t fr = 0, tot = 0;
        CUDA_OR_RETURN(cudaMemGetInfo(&fr, &tot));
        const size_t keep = (size_t)2 << 30;
        S->budget = fr > keep ? fr - keep : fr / 2;
    }
    *out = S.release();
    return EQD_OK;
}

// Stream priorities of a served grid: smaller grids get higher priority, so
// their short kernels take SM slots ahead of a large grid's long ones (a
// request on the h = 100 m grid is not starved by h = 25 m work). Within a
// grid the vector kernels stay one level above the stencil applies.
static int set_grid_priority(eqd_grid *G) {
    int least = 0, greatest = 0;
    CUDA_OR_RETURN(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    const double ntot = 6.0 * G->gc.n1 * G->gc.n2 * G->gc.n3;
    const int bucket = std::max(0, (int)std::floor(std::log10(std::max(ntot, 1.0))) - 4);  // 0: < 1e5 DOF
    const int step = least > greatest ? -1 : 1;                 // direction of "higher priority"
    const int span = std::abs(least - greatest);
    const int main_p = greatest - step * std::min(span, 1 + bucket);
    const int rest_p = greatest - step * std::min(span, bucket);
    CUDA_OR_RETURN(cudaStreamSynchronize(G->stream));
    for (cudaStream_t t : {G->stream, G->stream2, G->stream_hi, G->stream2_hi}) cudaStreamDestroy(t);
    CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream, cudaStreamNonBlocking, main_p));
    CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream2, cudaStreamNonBlocking, main_p));
    CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream_hi, cudaStreamNonBlocking, rest_p));
    CUDA_OR_RETURN(cudaStreamCreateWithPriority(&G->stream2_hi, cudaStreamNonBlocking, rest_p));
    G->ws.graph_key.clear();  // recapture on the new streams
    return EQD_OK;
}

extern "C" int eqd_server_add_grid(eqd_server *S, eqd_grid *G, int32_t slots) {
    if (!S || !G || slots < 0) return fail(EQD_ERR_ARG, "invalid argument");
    {
        std::lock_guard<std::mutex> lk(S->mu);
        for (auto &g : S->grids)
            if (g->G == G) return fail(EQD_ERR_ARG, "grid already attached");
    }
    std::lock_guard<std::mutex> glk(G->mtx);
    if (G->served) return fail(EQD_ERR_ARG, "the grid is attached to another server");
    CUDA_OR_RETURN(cudaSetDevice(G->desc.device));
    const GridConst &gc = G->gc;
    const int mixed = S->opts.precision == EQD_PREC_MIXED;
    Path path;
    int rc = mixed ? choose_path<float>(G, S->opts, false, false, path)
                   : choose_path<double>(G, S->opts, false, false, path);
    if (rc) return rc;
    auto bytes = [&]() {
        return mixed ? slot_bytes<float>(G, S->opts, false, path) : slot_bytes<double>(G, S->opts, false, path);
    };
    std::unique_ptr<SrvGrid> g(new SrvGrid());
    {
        std::lock_guard<std::mutex> lk(S->mu);
        const uint64_t left = S->budget > S->used ? S->budget - S->used : 0;
        if (path.xm && left / bytes() < (uint64_t)std::max(slots, 1)) path.xm = false;  // as resolve_chunk
        const size_t per_slot = bytes();
        const long long fit = (long long)(left / per_slot);
        const int want = slots > 0 ? slots : (int)std::min<long long>(fit, 512);
        if (want < 1 || (long long)want > fit)
            return fail(EQD_ERR_OOM, "the server's HBM budget has room for " + std::to_string(fit) +
                                         " slot(s) of this grid");
        g->slots = want;
        g->bytes = (size_t)want * per_slot;
        S->used += g->bytes;
    }
    g->G = G;
    rc = set_grid_priority(G);
    if (rc) {
        std::lock_guard<std::mutex> lk(S->mu);
        S->used -= g->bytes;
        return rc;
    }
    if (mixed) {
        g->r32.reset(new SlotRun<float>());
        rc = g->r32->setup(G, S->opts, g->slots, false, false, path);
    } else {
        g->r64.reset(new SlotRun<double>());
        rc = g->r64->setup(G, S->opts, g->slots, false, false, path);
    }
    if (!rc) {
        cudaError_t e = g->kstage.assign(2 * gc.nf * g->slots, 0.0);
        if (e != cudaSuccess) rc = fail(EQD_ERR_OOM, "pinned staging buffer");
    }
    if (!rc) {
        cudaError_t e = cudaStreamSynchronize(G->stream);
        if (e != cudaSuccess) rc = fail(EQD_ERR_CUDA, cudaGetErrorString(e));
    }
    if (rc) {
        std::lock_guard<std::mutex> lk(S->mu);
        S->used -= g->bytes;
        return rc;
    }
    G->served = true;
    std::lock_guard<std::mutex> lk(S->mu);
    SrvGrid *gp = g.get();
    S->grids.push_back(std::move(g));
    gp->worker = std::thread(grid_loop, S, gp);
    return EQD_OK;
}

extern "C" int eqd_server_submit(eqd_server *S, eqd_grid *G, const int32_t *cols, int32_t ncols, double *k_out,
                                 int64_t *request_id) {
    if (!S || !G || (!cols && ncols > 0) || ncols < 0 || (!k_out && ncols > 0) || !request_id)
        return fail(EQD_ERR_ARG, "invalid argument");
    if (ncols >= (1 << kTagBits)) return fail(EQD_ERR_ARG, "too many columns in one request");
    std::lock_guard<std::mutex> lk(S->mu);
    if (S->fatal) return fail(S->fatal, "server stopped: " + S->fatal_msg);
    SrvGrid *g = nullptr;
    for (auto &x : S->grids)
        if (x->G == G) g = x.get();
    if (!g) return fail(EQD_ERR_ARG, "grid not attached to this server");
    const int nf = G->gc.nf;
    for (int i = 0; i < ncols; ++i)
        if (cols[i] < 0 || cols[i] >= 2 * nf) return fail(EQD_ERR_ARG, "column index out of range");
    std::unique_ptr<SrvRequest> r(new SrvRequest());
    r->id = S->next_id++;
    r->k_out = k_out;
    r->ncols = r->remaining = ncols;
    r->t_submit = S->now();
    if (ncols == 0) {
        r->state = 2;
        r->t_start = r->t_done = r->t_submit;
    }
    for (int i = 0; i < ncols; ++i) {
        ColWork c;
        c.slip_node = cols[i] % nf;
        c.slip_comp = cols[i] / nf;
        c.tag = (r->id << kTagBits) | i;
        g->pending.push_back(c);
    }
    *request_id = r->id;
    S->reqs[r->id] = std::move(r);
    S->cv_work.notify_all();
    return EQD_OK;
}

static SrvRequest *find_req(eqd_server *S, int64_t id) {
    auto it = S->reqs.find(id);
    return it == S->reqs.end() ? nullptr : it->second.get();
}

extern "C" int eqd_server_wait(eqd_server *S, int64_t id, double timeout_s) {
    if (!S) return fail(EQD_ERR_ARG, "null server");
    std::unique_lock<std::mutex> lk(S->mu);
    SrvRequest *r = find_req(S, id);
    if (!r) return fail(EQD_ERR_ARG, "unknown request id");
    const auto pred = [&] { return r->state >= 2; };
    if (timeout_s < 0) S->cv_done.wait(lk, pred);
    else if (!S->cv_done.wait_for(lk, std::chrono::duration<double>(timeout_s), pred))
        return fail(EQD_ERR_TIMEOUT, "request not done within the timeout");
    if (r->state == 3) return fail(r->err, r->msg);
    return EQD_OK;
}

extern "C" int eqd_server_poll(eqd_server *S, int64_t id, int32_t *done) {
    if (!S || !done) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(S->mu);
    SrvRequest *r = find_req(S, id);
    if (!r) return fail(EQD_ERR_ARG, "unknown request id");
    *done = r->state >= 2;
    if (r->state == 3) return fail(r->err, r->msg);
    return EQD_OK;
}

extern "C" int eqd_server_request_info(eqd_server *S, int64_t id, eqd_request_info *info) {
    if (!S || !info) return fail(EQD_ERR_ARG, "invalid argument");
    std::lock_guard<std::mutex> lk(S->mu);
    SrvRequest *r = find_req(S, id);
    if (!r) return fail(EQD_ERR_ARG, "unknown request id");
    info->state = r->state;
    info->ncols = r->ncols;
    info->unconverged = r->unconverged;
    info->max_iterations = r->max_it;
    info->iterations = r->iterations;
    info->t_submit = r->t_submit;
    info->t_start = r->t_start;
    info->t_done = r->t_done;
    return EQD_OK;
}

extern "C" int eqd_server_release(eqd_server *S, int64_t id) {
    if (!S) return fail(EQD_ERR_ARG, "null server");
    std::lock_guard<std::mutex> lk(S->mu);
    SrvRequest *r = find_req(S, id);
    if (!r) return fail(EQD_ERR_ARG, "unknown request id");
    if (r->state < 2) return fail(EQD_ERR_ARG, "request still in flight");
    S->reqs.erase(id);
    return EQD_OK;
}

extern "C" int eqd_server_destroy(eqd_server *S) {
    if (!S) return EQD_OK;
    {
        std::lock_guard<std::mutex> lk(S->mu);
        S->stop = true;
    }
    S->cv_work.notify_all();
    for (auto &g : S->grids)
        if (g->worker.joinable()) g->worker.join();
    for (auto &g : S->grids) {
        cudaSetDevice(g->G->desc.device);
        cudaStreamSynchronize(g->G->stream);
        g->r32.reset();
        g->r64.reset();
        std::lock_guard<std::mutex> glk(g->G->mtx);
        g->G->served = false;
    }
    delete S;
    return EQD_OK;
}

// ---------------------------------------------------------------------------
// Time-loop right-hand side (eqd_rhs_*) and batched friction solves
// ---------------------------------------------------------------------------
struct eqd_rhs {
    int device = 0;
    int nf = 0;
    eqd_rhs_params p{};
    DevBuf K, dtau, io, ap_ptr, ap_idx, ap_val, source, active, vprev, tau, sigma_low, floor_nodes, floor_hits;
    PinnedArr<double> host;  // io's image: u, the status word, du
    cudaStream_t stream = nullptr;
};

static FrictionConst friction_const(const eqd_rhs_params &p) {
    return FrictionConst{p.a, p.b, p.Dc, p.V_star, p.f_star};
}

static bool newton_ok(const eqd_rhs_params &p) {
    return p.newton_tol > 0 && p.newton_maxiter > 0 && p.newton_maxstep > 0 && p.a > 0 && p.Dc > 0 && p.V_star > 0;
}

extern "C" int eqd_rhs_create(int32_t device, int32_t nf, const double *K, const eqd_rhs_params *params,
                              const int32_t *ap_ptr, const int32_t *ap_idx, const double *ap_val, const double *source,
                              const uint8_t *active, eqd_rhs **out) {
    if (!out || !K || !params || nf < 1 || !ap_ptr || (!ap_idx && ap_ptr[nf] > 0) || (!ap_val && ap_ptr[nf] > 0))
        return fail(EQD_ERR_ARG, "invalid argument");
    *out = nullptr;
    if (!newton_ok(*params)) return fail(EQD_ERR_ARG, "invalid friction or Newton parameters");
    if (params->injection == 1 && (params->well_cell < 0 || params->well_cell >= nf))
        return fail(EQD_ERR_ARG, "well_cell out of range");
    const int nnz = ap_ptr[nf];
    for (int i = 0; i < nf; ++i)
        if (ap_ptr[i + 1] < ap_ptr[i]) return fail(EQD_ERR_ARG, "Ap row pointers must be non-decreasing");
    for (int k = 0; k < nnz; ++k)
        if (ap_idx[k] < 0 || ap_idx[k] >= nf) return fail(EQD_ERR_ARG, "Ap column index out of range");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
    if (device < 0 || device >= ndev) return fail(EQD_ERR_ARG, "device ordinal out of range");
    CUDA_OR_RETURN(cudaSetDevice(device));
    std::unique_ptr<eqd_rhs> R(new eqd_rhs());
    R->device = device;
    R->nf = nf;
    R->p = *params;
    const long long n = 2LL * nf;
    CUDA_OR_RETURN(cudaStreamCreateWithFlags(&R->stream, cudaStreamNonBlocking));
    CUDA_OR_RETURN(R->K.ensure(sizeof(double) * n * n));
    CUDA_OR_RETURN(R->dtau.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(R->io.ensure(sizeof(double) * (8LL * nf + 3)));
    CUDA_OR_RETURN(R->host.assign(8 * nf + 3, 0.0));
    CUDA_OR_RETURN(R->ap_ptr.ensure(sizeof(int) * (nf + 1)));
    CUDA_OR_RETURN(R->ap_idx.ensure(sizeof(int) * std::max(nnz, 1)));
    CUDA_OR_RETURN(R->ap_val.ensure(sizeof(double) * std::max(nnz, 1)));
    CUDA_OR_RETURN(R->source.ensure(sizeof(double) * nf));
    CUDA_OR_RETURN(R->active.ensure(nf));
    CUDA_OR_RETURN(R->vprev.ensure(sizeof(double) * nf));
    CUDA_OR_RETURN(R->tau.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(R->sigma_low.ensure(sizeof(double) * nf));
    CUDA_OR_RETURN(R->floor_nodes.ensure(nf));
    CUDA_OR_RETURN(R->floor_hits.ensure(sizeof(unsigned long long)));
    cudaStream_t st = R->stream;
    CUDA_OR_RETURN(cudaMemcpyAsync(R->K.p, K, sizeof(double) * n * n, cudaMemcpyHostToDevice, st));
    CUDA_OR_RETURN(cudaMemcpyAsync(R->ap_ptr.p, ap_ptr, sizeof(int) * (nf + 1), cudaMemcpyHostToDevice, st));
    if (nnz > 0) {
        CUDA_OR_RETURN(cudaMemcpyAsync(R->ap_idx.p, ap_idx, sizeof(int) * nnz, cudaMemcpyHostToDevice, st));
        CUDA_OR_RETURN(cudaMemcpyAsync(R->ap_val.p, ap_val, sizeof(double) * nnz, cudaMemcpyHostToDevice, st));
    }
    if (source) CUDA_OR_RETURN(cudaMemcpyAsync(R->source.p, source, sizeof(double) * nf, cudaMemcpyHostToDevice, st));
    else CUDA_OR_RETURN(cudaMemsetAsync(R->source.p, 0, sizeof(double) * nf, st));
    if (active) CUDA_OR_RETURN(cudaMemcpyAsync(R->active.p, active, nf, cudaMemcpyHostToDevice, st));
    else CUDA_OR_RETURN(cudaMemsetAsync(R->active.p, 1, nf, st));
    std::vector<double> init(nf, 1e-12), low(nf, INFINITY);
    CUDA_OR_RETURN(cudaMemcpyAsync(R->vprev.p, init.data(), sizeof(double) * nf, cudaMemcpyHostToDevice, st));
    CUDA_OR_RETURN(cudaMemcpyAsync(R->sigma_low.p, low.data(), sizeof(double) * nf, cudaMemcpyHostToDevice, st));
    CUDA_OR_RETURN(cudaMemsetAsync(R->floor_nodes.p, 0, nf, st));
    CUDA_OR_RETURN(cudaMemsetAsync(R->floor_hits.p, 0, sizeof(unsigned long long), st));
    CUDA_OR_RETURN(cudaMemsetAsync(R->tau.p, 0, sizeof(double) * n, st));
    CUDA_OR_RETURN(cudaStreamSynchronize(st));
    *out = R.release();
    return EQD_OK;
}

extern "C" int eqd_rhs_eval(eqd_rhs *R, double t, const double *u, double *du) {
    if (!R || !u || !du) return fail(EQD_ERR_ARG, "invalid argument");
    CUDA_OR_RETURN(cudaSetDevice(R->device));
    const int nf = R->nf;
    const long long nu = 4LL * nf + (R->p.injection == 1 ? 1 : 0);
    const long long n = 2LL * nf;
    cudaStream_t st = R->stream;
    // One copy each way, through page-locked memory: u and a zero status word
    // in, the status and du out.
    double *hu = R->host.data(), *du_dev = R->io.as<double>() + nu + 1;
    std::memcpy(hu, u, sizeof(double) * nu);
    hu[nu] = 0.0;
    CUDA_OR_RETURN(cudaMemcpyAsync(R->io.p, hu, sizeof(double) * (nu + 1), cudaMemcpyHostToDevice, st));
    CUDA_OR_RETURN(launch_gemv(st, R->K.as<double>(), R->io.as<double>(), (int)n, 1, R->dtau.as<double>()));
    RhsParams P{};
    P.fr = friction_const(R->p);
    P.sigma0 = R->p.sigma0;
    P.sigma_min = R->p.sigma_min;
    P.eta = R->p.eta;
    P.tau0_2 = R->p.tau0_2;
    P.tau0_3 = R->p.tau0_3;
    P.src_scale = t < R->p.t_off ? R->p.q0 / (R->p.beta * R->p.phi) : 0.0;
    P.tol = R->p.newton_tol;
    P.maxstep = R->p.newton_maxstep;
    P.maxiter = R->p.newton_maxiter;
    P.nf = nf;
    P.peaceman = R->p.injection == 1;
    P.well_cell = R->p.well_cell;
    P.WI = R->p.WI;
    P.S_e = R->p.S_e;
    P.S_well = R->p.S_well;
    P.Qinj = t < R->p.t_off ? R->p.Q0 : 0.0;
    rhs_node_kernel<<<(unsigned)((nf + 127) / 128), 128, 0, st>>>(
        P, R->dtau.as<double>(), R->io.as<double>(), du_dev, R->ap_ptr.as<int>(), R->ap_idx.as<int>(),
        R->ap_val.as<double>(), R->source.as<double>(), R->active.as<unsigned char>(), R->vprev.as<double>(),
        R->tau.as<double>(), R->sigma_low.as<double>(), R->floor_nodes.as<unsigned char>(),
        R->floor_hits.as<unsigned long long>(), reinterpret_cast<unsigned *>(du_dev - 1));
    CUDA_OR_RETURN(cudaGetLastError());
    CUDA_OR_RETURN(cudaMemcpyAsync(hu + nu, du_dev - 1, sizeof(double) * (nu + 1), cudaMemcpyDeviceToHost, st));
    CUDA_OR_RETURN(cudaStreamSynchronize(st));
    unsigned h = 0;
    std::memcpy(&h, hu + nu, sizeof(h));
    std::memcpy(du, hu + nu + 1, sizeof(double) * nu);
    if (h & RHS_NEWTON_FAILED)
        return fail(EQD_ERR_NOT_CONVERGED, "solve_slip_rate did not converge at some fault node");
    return EQD_OK;
}

extern "C" int eqd_rhs_fields(eqd_rhs *R, double *tau, double *vprev) {
    if (!R) return fail(EQD_ERR_ARG, "invalid argument");
    CUDA_OR_RETURN(cudaSetDevice(R->device));
    if (tau)
        CUDA_OR_RETURN(cudaMemcpyAsync(tau, R->tau.p, sizeof(double) * 2 * R->nf, cudaMemcpyDeviceToHost, R->stream));
    if (vprev)
        CUDA_OR_RETURN(cudaMemcpyAsync(vprev, R->vprev.p, sizeof(double) * R->nf, cudaMemcpyDeviceToHost, R->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(R->stream));
    return EQD_OK;
}

extern "C" int eqd_rhs_report(eqd_rhs *R, double *sigma_lowest, int64_t *floor_hits, int32_t *floor_nodes) {
    if (!R) return fail(EQD_ERR_ARG, "invalid argument");
    CUDA_OR_RETURN(cudaSetDevice(R->device));
    std::vector<double> low(R->nf);
    std::vector<unsigned char> fn(R->nf);
    unsigned long long hits = 0;
    CUDA_OR_RETURN(cudaMemcpyAsync(low.data(), R->sigma_low.p, sizeof(double) * R->nf, cudaMemcpyDeviceToHost, R->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(fn.data(), R->floor_nodes.p, R->nf, cudaMemcpyDeviceToHost, R->stream));
    CUDA_OR_RETURN(cudaMemcpyAsync(&hits, R->floor_hits.p, sizeof(hits), cudaMemcpyDeviceToHost, R->stream));
    CUDA_OR_RETURN(cudaStreamSynchronize(R->stream));
    double m = INFINITY;
    int cnt = 0;
    for (int i = 0; i < R->nf; ++i) {
        m = std::min(m, low[i]);
        cnt += fn[i] != 0;
    }
    if (sigma_lowest) *sigma_lowest = m;
    if (floor_hits) *floor_hits = (int64_t)hits;
    if (floor_nodes) *floor_nodes = cnt;
    return EQD_OK;
}

extern "C" int eqd_rhs_destroy(eqd_rhs *R) {
    if (!R) return EQD_OK;
    cudaSetDevice(R->device);
    if (R->stream) {
        cudaStreamSynchronize(R->stream);
        cudaStreamDestroy(R->stream);
    }
    delete R;
    return EQD_OK;
}

extern "C" int eqd_friction_solve(int32_t device, int32_t n, const double *T, const double *theta, const double *sigma,
                                  double eta, const eqd_rhs_params *params, const double *V0, double *V) {
    if (n < 0 || (n > 0 && (!T || !theta || !sigma || !V)) || !params) return fail(EQD_ERR_ARG, "invalid argument");
    if (!newton_ok(*params)) return fail(EQD_ERR_ARG, "invalid friction or Newton parameters");
    if (n == 0) return EQD_OK;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(EQD_ERR_NO_DEVICE, "no CUDA device visible");
    if (device < 0 || device >= ndev) return fail(EQD_ERR_ARG, "device ordinal out of range");
    CUDA_OR_RETURN(cudaSetDevice(device));
    DevBuf dT, dth, dsg, dv0, dV, dst;
    CUDA_OR_RETURN(dT.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(dth.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(dsg.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(dV.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(dst.ensure(sizeof(unsigned)));
    if (V0) CUDA_OR_RETURN(dv0.ensure(sizeof(double) * n));
    CUDA_OR_RETURN(cudaMemcpy(dT.p, T, sizeof(double) * n, cudaMemcpyHostToDevice));
    CUDA_OR_RETURN(cudaMemcpy(dth.p, theta, sizeof(double) * n, cudaMemcpyHostToDevice));
    CUDA_OR_RETURN(cudaMemcpy(dsg.p, sigma, sizeof(double) * n, cudaMemcpyHostToDevice));
    if (V0) CUDA_OR_RETURN(cudaMemcpy(dv0.p, V0, sizeof(double) * n, cudaMemcpyHostToDevice));
    CUDA_OR_RETURN(cudaMemset(dst.p, 0, sizeof(unsigned)));
    friction_solve_kernel<<<(unsigned)((n + 127) / 128), 128>>>(
        n, dT.as<double>(), dth.as<double>(), dsg.as<double>(), eta, friction_const(*params),
        V0 ? dv0.as<double>() : nullptr, params->newton_tol, params->newton_maxiter, params->newton_maxstep,
        dV.as<double>(), dst.as<unsigned>());
    CUDA_OR_RETURN(cudaGetLastError());
    unsigned h = 0;
    CUDA_OR_RETURN(cudaMemcpy(V, dV.p, sizeof(double) * n, cudaMemcpyDeviceToHost));
    CUDA_OR_RETURN(cudaMemcpy(&h, dst.p, sizeof(unsigned), cudaMemcpyDeviceToHost));
    if (h & RHS_NEWTON_FAILED)
        return fail(EQD_ERR_NOT_CONVERGED, "solve_slip_rate failed to converge");
    return EQD_OK;
}
