// Resident CG: many iterations of one column's CG inside one launch, the
// column's vectors held on chip by a cluster of CTAs.
//
// The streamed iteration moves a column's vectors eleven times through HBM
// and pays four to seven launches; on a small grid neither the march's few
// CTAs nor the launches fill the device (one column at h = 50 m: 98 us an
// iteration, 60 us of it the three-CTA apply). Here a cluster of M CTAs owns
// one column: p (with its halo) and two of the three stress sums F live in
// shared memory, r, the solution and q in registers, so an iteration touches
// no global memory; a line's new p is stored straight into the shared memory
// of the CTAs that have it in their halo, dot products are exchanged the same
// way, and two cluster barriers order an iteration. The kernel ends when the
// column needs its FP64 true residual (mixed precision), is done (FP64), or
// has run kmax iterations.
//
// Operator (plane_march.cuh has the reference citations), per side:
//   G_k = D1_k v_k,  F_j = lam G_j + (lam + mu) sum_{k != j} G_k,
//   w_j = mu (sum_a D2_a + D2_j) v_j + D1_j F_j,
// which needs only five-point (closure: six-point) rows; w then gets the SAT
// terms at x = 0, P and -H.
//
// A thread owns half a line (x1 points of one node and side): its x1
// derivatives come from registers with coefficients from the kernel's
// parameters (n1 is compiled in, so every closure row is straight code), and
// the two sides of a line sit in adjacent lanes, so a fault node's sides
// exchange by one shuffle. The x2 and x3 rows take their coefficients and the
// places of their outer points from a table by the line's row class: interior
// and closure rows run the same code, with the same number of loads. All that
// reads p is done in one pass (F and the second derivatives share loads); the
// F terms follow after a barrier.
// Whole lines per thread left an SM four warps (19 k clocks an iteration at
// 17 x 17 x 9 on four CTAs, against 11 k); one component of a line per thread
// gave it 24 but 34 % more instructions.
//
// What bounds it: latency at 16 warps an SM (the two cluster barriers, the
// stores to the neighbours, the FP64 reduction), then shared-memory wavefronts
// (about 45 a point). Measured against the streamed iteration: one column at
// h = 50 m 15 us an iteration (was 98), one slip's traction 2.2 ms (14.5), the
// ten Toeplitz columns 3.2 ms (15.7), three columns at h = 100 m 1.6 ms (8.5),
// all 578 there 9 ms (34), all 2,178 at h = 50 m 212 ms (300), where the host
// does not hold a call up.
//
// FP64 lines of more than 13 points take smaller tiles and more parts a line:
// one column at 17^3 1.8 ms (streamed 14), 96 at 19^3 33 ms (48), 200 at 17^3
// 19 ms (41). A grid that no cluster holds (GRID) is shared by a team of CTAs
// of one cooperative launch, which exchange p and the dot products through
// global memory (L2) and meet at a counter there; each team takes columns in
// turn. One right-hand side at 25^3 on 49 CTAs: 20 us an iteration, 5.3 ms
// (streamed 22 to 27: four launches of 7 to 57 us an iteration on a few CTAs).
//
// The order of every sum is fixed by the plan, which depends on the grid and
// the precision only: a column gives the same bits alone and in any batch.
// (Explicit right-hand sides on grids of a team that is for a few of them: while
// a call has no more than four a team; beyond that it streams them.)
#pragma once
#include <type_traits>

#include "resident_plan.h"
#include "solver_kernels.cuh"

namespace eqd {

template <typename T>
struct ResCoef {
    T lam, lpm, sat, mu, mu2;        // mu2 = 2 mu
    T dlo[4];                        // boundary derivative
};

struct ResTables {
    const ResRank *ranks;
    const int *chunks;
    const ResLine *lines;
    const int *gofs;
    const int *push;
    const ResPull *pull;
    const void *tab;  // fill_res_tables rows, T
    const int *off;
};

template <typename T>
__host__ __device__ __forceinline__ void res_load4(const T *t, T (&c)[4]) {
#ifdef __CUDA_ARCH__
    if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(t);
        c[0] = v.x, c[1] = v.y, c[2] = v.z, c[3] = v.w;
    } else {
        const double2 v = reinterpret_cast<const double2 *>(t)[0], w = reinterpret_cast<const double2 *>(t)[1];
        c[0] = v.x, c[1] = v.y, c[2] = w.x, c[3] = w.y;
    }
#else
    for (int k = 0; k < 4; ++k) c[k] = t[k];
#endif
}

// The rows of one line on one axis: fill_res_tables' layout.
template <typename T>
struct ResLineRow {
    const T *t;
    const int *o;
};

// Row x of an x1 operator on a line held in registers (zero entries skipped).
template <bool SECOND, int N1, typename T>
__host__ __device__ __forceinline__ T res_x1_dot(const T (&c)[N1][6], const T (&l)[N1], int x) {
    T s = T(0);
    bool any = false;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (!res_nz(SECOND, x, N1, k)) continue;
        const T t = l[res_start(x, N1) + k];
        s = any ? s + c[x][k] * t : c[x][k] * t;
        any = true;
    }
    return s;
}

// The first derivatives at the points [XA, XB) of a line whose p starts at v
// (side included). put(x, G1, G2, G3).
template <typename T, int N1, typename G, int XA, int XB, typename PUT>
__host__ __device__ __forceinline__ void res_line_grad(const ResX1<T, N1> &X, const T *v, T sgn, ResLineRow<T> row2,
                                                        ResLineRow<T> row3, PUT put) {
    constexpr int LO = res_start(XA, N1), HI = res_start(XB - 1, N1) + 6;
    T l[N1];
#pragma unroll
    for (int x = 0; x < N1; ++x) l[x] = x >= LO && x < HI && x < N1 - 1 ? v[x * G::PSZ] : T(0);  // p is 0 at N1 - 1
    T c2[4], c3[4];
    res_load4(row2.t, c2);
    res_load4(row3.t, c3);
    int o2[4], o3[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        o2[k] = row2.o[k] + G::CS;
        o3[k] = row3.o[k] * G::R2 + 2 * G::CS;
    }
#pragma unroll
    for (int x = XA; x < XB; ++x) {
        const T G1 = sgn * res_x1_dot<false>(X.c1, l, x);
        T G2 = T(0), G3 = T(0);
        if (x < N1 - 1) {
            const T *vx = v + x * G::PSZ;
            G2 = c2[0] * vx[o2[0]];
            G3 = c3[0] * vx[o3[0]];
#pragma unroll
            for (int k = 1; k < 4; ++k) {
                G2 += c2[k] * vx[o2[k]];
                G3 += c3[k] * vx[o3[k]];
            }
        }
        put(x, G1, G2, G3);
    }
}

// All that an own line's points [XA, XB) need of p: F there (putf(x, F1, F2,
// F3); x = N1-1 has F1 only), the second derivatives w, the points' p itself,
// and, where the points start at the fault, the traction on the fixed +x1 axis
// there. v: the line's p, component 1.
template <typename T, int N1, typename G, int XA, int XB, int W, typename PUTF>
__host__ __device__ __forceinline__ void res_own_p(const ResCoef<T> &C, const ResX1<T, N1> &X, const T *v, T sgn,
                                                   ResLineRow<T> row2, ResLineRow<T> row3, T (&w)[W][3],
                                                   T (&pv)[W][3], T (&tau)[3], PUTF putf) {
    static_assert(W >= XB - XA, "a place for every point");
    constexpr int XE = XB == N1 - 1 ? N1 : XB;  // the last half also has F1 at the far field
    constexpr int LO = res_start(XA, N1), HI = res_start(XE - 1, N1) + 6;
    const int oa2 = row2.o[0], ob2 = row2.o[3], oa3 = row3.o[0] * G::R2, ob3 = row3.o[3] * G::R2;
    T c2[4], c3[4], s2[4], s3[4];  // D1; mu D2: outer, -1, own, +1, and the other outer
    res_load4(row2.t, c2);
    res_load4(row3.t, c3);
    res_load4(row2.t + 4, s2);
    res_load4(row3.t + 4, s3);
    const T s24 = row2.t[8], s34 = row3.t[8];
    T G1[XE - XA], G2[XB - XA], G3[XB - XA], dh[3], d2 = T(0), d3 = T(0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const T *u = v + j * G::CS;
        T l[N1];
#pragma unroll
        for (int x = 0; x < N1; ++x) l[x] = x >= LO && x < HI && x < N1 - 1 ? u[x * G::PSZ] : T(0);  // p is 0 at N1 - 1
#pragma unroll
        for (int x = XA; x < XB; ++x) {
            const T *ux = u + x * G::PSZ;
            const T a2 = ux[oa2], m2 = ux[-1], p2 = ux[1], b2 = ux[ob2];
            const T a3 = ux[oa3], m3 = ux[-G::R2], p3 = ux[G::R2], b3 = ux[ob3];
            const T x1 = res_x1_dot<true>(X.c2, l, x);
            const T x2 = s2[0] * a2 + s2[1] * m2 + s2[2] * l[x] + s2[3] * p2 + s24 * b2;
            const T x3 = s3[0] * a3 + s3[1] * m3 + s3[2] * l[x] + s3[3] * p3 + s34 * b3;
            w[x - XA][j] = (j == 0 ? x1 + x1 : x1) + (j == 1 ? x2 + x2 : x2) + (j == 2 ? x3 + x3 : x3);
            pv[x - XA][j] = l[x];
            if (j == 1) G2[x - XA] = c2[0] * a2 + c2[1] * m2 + c2[2] * p2 + c2[3] * b2;
            if (j == 2) G3[x - XA] = c3[0] * a3 + c3[1] * m3 + c3[2] * p3 + c3[3] * b3;
            if (j == 0 && x == 0) {
                d2 = c2[0] * a2 + c2[1] * m2 + c2[2] * p2 + c2[3] * b2;
                d3 = c3[0] * a3 + c3[1] * m3 + c3[2] * p3 + c3[3] * b3;
            }
        }
        if (j == 0) {
#pragma unroll
            for (int x = XA; x < XE; ++x) G1[x - XA] = sgn * res_x1_dot<false>(X.c1, l, x);
        }
        if (XA == 0) {
            T s = C.dlo[0] * l[0];
#pragma unroll
            for (int k = 1; k < 4; ++k) s += C.dlo[k] * l[k];
            dh[j] = sgn * s;
        }
    }
#pragma unroll
    for (int x = XA; x < XE; ++x) {
        const T g1 = G1[x - XA], g2 = x < XB ? G2[x < XB ? x - XA : 0] : T(0), g3 = x < XB ? G3[x < XB ? x - XA : 0] : T(0);
        putf(x, C.lam * g1 + C.lpm * (g2 + g3), C.lam * g2 + C.lpm * (g1 + g3), C.lam * g3 + C.lpm * (g1 + g2));
    }
    if (XA == 0) {
        tau[0] = C.lam * (G1[0] + G2[0] + G3[0]) + C.mu2 * dh[0];
        tau[1] = C.mu * (d2 + dh[1]);
        tau[2] = C.mu * (d3 + dh[2]);
    }
}

// The F terms of w at the points [XA, XB) of an own line. f1: the line's F1
// (stride f1s); f2, f3: its places in F2 and F3 (side included).
template <typename T, int N1, typename G, int XA, int XB, int W>
__host__ __device__ __forceinline__ void res_own_f(const ResX1<T, N1> &X, const T *f1, int f1s, const T *f2,
                                                   const T *f3, T sgn, ResLineRow<T> row2, ResLineRow<T> row3,
                                                   T (&w)[W][3]) {
    constexpr int LO = res_start(XA, N1), HI = res_start(XB - 1, N1) + 6;
    const int oa2 = row2.o[0], ob2 = row2.o[3], oa3 = row3.o[0] * G::R2b, ob3 = row3.o[3] * G::R2b;
    T c2[4], c3[4];
    res_load4(row2.t, c2);
    res_load4(row3.t, c3);
    T l[N1];
#pragma unroll
    for (int x = 0; x < N1; ++x) l[x] = x >= LO && x < HI ? f1[x * f1s] : T(0);
#pragma unroll
    for (int x = XA; x < XB; ++x) {
        const T *g2 = f2 + x * G::PSa, *g3 = f3 + x * G::PSb;
        T(&o)[3] = w[x - XA];
        o[0] += sgn * res_x1_dot<false>(X.c1, l, x);
        o[1] += c2[0] * g2[oa2] + c2[1] * g2[-1] + c2[2] * g2[1] + c2[3] * g2[ob2];
        o[2] += c3[0] * g3[oa3] + c3[1] * g3[-G::R2b] + c3[2] * g3[G::R2b] + c3[3] * g3[ob3];
    }
}

template <typename T>
inline ResCoef<T> res_coef(double h1, double lam, double mu, double sat) {
    ResCoef<T> C{};
    C.lam = (T)lam;
    C.lpm = (T)(lam + mu);
    C.sat = (T)sat;
    C.mu = (T)mu;
    C.mu2 = (T)(2 * mu);
    for (int k = 0; k < 4; ++k) C.dlo[k] = (T)(kDb[k].v() / h1);
    return C;
}

// Threads of an instance at most: 512 x 128 registers, or 256 x 255 where a
// thread's part of a line needs them.
template <typename T, int N1, int NP>
constexpr int res_max_threads() {
    return (int)sizeof(T) / 4 * (N1 - 1) / NP <= 5 ? 32 * kResMaxWarps : 16 * kResMaxWarps;
}

// A team of CTAs of a cooperative launch: its copy of p, its partial sums, and
// the counter that it meets at.
template <typename T>
struct ResTeam {
    T *p;             // [team][rank][3 CS]
    double *red;      // [team][rank][8]
    unsigned *count;  // [team][32], its first zero at launch
    int teams;
    unsigned *err;
};

// Every thread of every CTA of the team: what they wrote before is seen by all
// after. False when the others have not come within about 2 s (recorded).
__device__ __forceinline__ bool team_barrier(unsigned *count, unsigned target, unsigned *err) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(count, 1u);
        unsigned long long t0 = 0;
        for (int i = 0;; ++i) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if ((int)(v - target) >= 0) break;
            if (i == 64) t0 = global_ns();
            if (i > 64 && ((i & 63) == 0) && global_ns() - t0 > 2000000000ull) {
                atomicOr(err, DERR_MBAR_TIMEOUT);
                ok = false;
                break;
            }
        }
    }
    return __syncthreads_and(ok);
}

// f(integral_constant<int, part>) for a run-time part of NP.
template <int NP, int P = 0, typename F>
__device__ __forceinline__ void res_with_part(int part, F &&f) {
    if constexpr (P + 1 < NP) {
        if (part != P) return res_with_part<NP, P + 1>(part, f);
    }
    f(std::integral_constant<int, P>());
}

// ---------------------------------------------------------------------------
// One column per cluster of d.M CTAs (grid: ncols * d.M CTAs, 32 NP d.nch0max
// threads each), or, GRID, team.teams teams of d.M CTAs that share the ncols
// columns (more warps there may take halo rows only). NP: parts of a line, one thread each. x: the FP32 correction of
// mixed precision, or the FP64 solution. On entry the direction is
// p = r + beta p.
// ---------------------------------------------------------------------------
template <typename T, int N1, int T2, int T3, int NP, bool GRID>
__global__ void __launch_bounds__((res_max_threads<T, N1, NP>()), 1)
resident_cg_kernel(const __grid_constant__ ResCoef<T> C, const __grid_constant__ ResX1<T, N1> X,
                   const __grid_constant__ ResDims d, ResTables tb, T *__restrict__ x_, T *__restrict__ r_,
                   T *__restrict__ p_, ColState st, SolveParams sp, int mixed, int kmax, int ncols, ResTeam<T> team) {
    using G = ResGeo<(int)sizeof(T), N1, T2, T3>;
    constexpr int NX = N1 - 1, XH = (NX + NP - 1) / NP;  // p is zero at the far field x = N1 - 1
    static_assert((NP - 1) * XH < NX, "every part of a line has points");
    constexpr bool ragged = NX % NP != 0;  // the last part has fewer
    const int M = d.M;
    const int tm = blockIdx.x / M;
    if (!GRID && st.status[tm] != COL_ACTIVE) return;  // the whole cluster: no barrier has been reached
    const int rank = GRID ? blockIdx.x % M : M > 1 ? cluster_rank() : 0;
    const ResRank R = tb.ranks[rank];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, nwarp = nthr >> 5;

    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *p = reinterpret_cast<T *>(smem_raw);
    T *F1 = reinterpret_cast<T *>(smem_raw + G::oF1);
    T *F2 = reinterpret_cast<T *>(smem_raw + G::oF2);
    T *F3 = reinterpret_cast<T *>(smem_raw + G::oF3);
    T *tab = reinterpret_cast<T *>(smem_raw + G::oTab);  // x2 row classes, then x3
    int *off = reinterpret_cast<int *>(smem_raw + G::oOff);
    double *red = reinterpret_cast<double *>(smem_raw + G::oRed);  // [rank][8], [warp][8], then alpha, beta, stop, sure
    double *wred = red + kResMaxTeam * 8;
    volatile double *step = wred + kResMaxWarps * 8;
    ResLine *lines = reinterpret_cast<ResLine *>(smem_raw + G::oLine);
    int *chunks = reinterpret_cast<int *>(smem_raw + G::oChunk);
    int *push = reinterpret_cast<int *>(smem_raw + G::oPush);

    // Tables, and zeros everywhere else (the far-field entries of p stay zero).
    for (int i = tid; i < G::oTab / (int)sizeof(T); i += nthr) p[i] = T(0);
    for (int i = tid; i < 18 * kResRow; i += nthr) tab[i] = static_cast<const T *>(tb.tab)[i];
    for (int i = tid; i < 18 * 4; i += nthr) off[i] = tb.off[i];
    for (int i = tid; i < R.nch * kResLinesPerChunk; i += nthr)
        lines[i] = tb.lines[R.chunk0 * kResLinesPerChunk + i];
    for (int i = tid; i < R.nch; i += nthr) chunks[i] = tb.chunks[R.chunk0 + i];
    for (int i = tid; i < R.nch0 * kResLinesPerChunk * d.npush; i += nthr) push[i] = tb.push[R.push0 * d.npush + i];
    for (int i = tid; i < (kResMaxTeam + kResMaxWarps + 1) * 8; i += nthr) red[i] = 0.0;
    __syncthreads();

    // This thread's part of a line: warps NP c .. NP c + NP - 1 have the CTA's own chunk c.
    const int side = lane & 1, sub = lane >> 1, chunk = warp / NP, half = warp % NP;
    const T sgn = side ? T(1) : T(-1);
    const bool has = chunk < R.nch0;
    ResLine L{};
    if (has) L = lines[chunk * kResLinesPerChunk + sub];
    const bool own = has && (L.info >> 8 & 1);
    const int npt = ragged && half == NP - 1 ? NX - (NP - 1) * XH : XH;  // this thread's points
    auto live = [&](int x) { return !ragged || x < npt; };
    auto rows = [&](int cls) { return ResLineRow<T>{tab + cls * kResRow, off + cls * 4}; };
    const ResLineRow<T> row2 = rows(L.info & 15), row3 = rows(9 + (L.info >> 4 & 15));
    T *const line = p + side * G::SS + L.plo;
    T *const mine = line + half * XH * G::PSZ;  // the own points of p
    T *const f1 = F1 + chunk * 32 + lane, *const f2 = F2 + side * G::SSa + L.f2, *const f3 = F3 + side * G::SSb + L.f3;
    const int f1s = R.nch0 * 32;
    const T hw23 = own ? row2.t[9] * row3.t[9] : T(0);
    const int cstr = d.n3 * d.PS, gstep = side ? 1 : -1;
    const int gline = 3 * side * cstr + (own ? tb.gofs[(R.chunk0 + chunk) * kResLinesPerChunk + sub] : 0) +
                      (side ? half * XH : NX - half * XH);
    T *const shared_p = GRID ? team.p + ((long long)tm * M + rank) * 3 * G::CS : nullptr;  // this CTA's part of the team's p
    const T *const team_p = GRID ? team.p + (long long)tm * M * 3 * G::CS : nullptr;
    double *const team_red = GRID ? team.red + (long long)tm * M * 8 : nullptr;
    unsigned met = 0;  // GRID: barriers passed

    // Everybody's p, or everybody's sums, are in place.
    auto meet = [&]() -> bool {
        if constexpr (GRID) {
            met += (unsigned)M;
            return team_barrier(team.count + 32 * tm, met, team.err);
        } else {
            if (M > 1) cluster_barrier();
            else __syncthreads();
            return true;
        }
    };

    for (int slot = tm; slot < ncols; slot += GRID ? team.teams : ncols) {
    if (GRID && st.status[slot] != COL_ACTIVE) continue;
    const long long g0 = (long long)slot * d.colstride + gline;
    T r[XH][3], xs[XH][3];
    double gamma = 0.0;
    double beta = st.beta[slot];
    const double tol = st.tol[slot], rr_ref = mixed ? st.rr_ref[slot] : 0.0;
    const long long itmax = sp.itmax > 0 ? sp.itmax : 2 * sp.ntot;
    int iters = st.iters[slot];

    // The new p of the own points: into its own place and into the halo of
    // every CTA that reads it. Those CTAs have left their last read of the
    // old value (the exchange of the dot products, or the barrier below).
    auto put_p = [&](const T (&v)[XH][3]) {
        if (!own) return;
#pragma unroll
        for (int x = 0; x < XH; ++x)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                if (live(x)) mine[x * G::PSZ + c * G::CS] = v[x][c];
        if constexpr (GRID) {
            T *out = shared_p + (mine - p);
#pragma unroll
            for (int x = 0; x < XH; ++x)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (live(x)) __stcg(out + x * G::PSZ + c * G::CS, v[x][c]);
            return;
        }
        const int *to = push + (chunk * kResLinesPerChunk + sub) * d.npush;
        for (int k = 0; k < d.npush; ++k) {
            const int w = to[k];
            if (w == -1) continue;
            T *q = map_cluster(p + side * G::SS + half * XH * G::PSZ, (int)((unsigned)w >> 28)) + (w & 0xffffff);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (!(w >> (24 + c) & 1)) continue;
#pragma unroll
                for (int x = 0; x < XH; ++x)
                    if (live(x)) q[x * G::PSZ + c * G::CS] = v[x][c];
            }
        }
    };

    if (!GRID && M > 1) cluster_barrier();  // every CTA's p is zeroed before its neighbours store into it
    {
        const T b = (T)beta;
        T v[XH][3];
#pragma unroll
        for (int x = 0; x < XH; ++x)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long g = g0 + c * (long long)cstr + x * gstep;
                const bool at = own && live(x);
                r[x][c] = at ? r_[g] : T(0);
                xs[x][c] = at ? x_[g] : T(0);
                v[x][c] = at ? r[x][c] + b * p_[g] : T(0);
            }
        put_p(v);
    }

    int status = COL_ACTIVE, flag = 0;
    for (int k = 0;; ++k) {
        if (!meet()) return;  // every CTA has its new p (clusters: halo included)
        if constexpr (GRID) {
            // The halo, from the team's copy: a lane per line and component, a
            // warp per plane, up to 32 loads in flight a thread.
            const ResPull *pl = tb.pull + R.pull0;
            constexpr int UE = 4, UP = 32 / sizeof(T);
            for (int e0 = lane; e0 < R.npull; e0 += 32 * UE) {
                ResPull q[UE];
#pragma unroll
                for (int u = 0; u < UE; ++u) q[u] = pl[min(e0 + 32 * u, R.npull - 1)];
                for (int s0 = warp; s0 < 2 * NX; s0 += UP * nwarp) {
                    T v[UE][UP];
#pragma unroll
                    for (int w = 0; w < UP; ++w) {
                        const int s = s0 + w * nwarp, o = s < NX ? s * G::PSZ : G::SS + (s - NX) * G::PSZ;
#pragma unroll
                        for (int u = 0; u < UE; ++u)
                            if (s < 2 * NX && e0 + 32 * u < R.npull) v[u][w] = __ldcg(team_p + q[u].src + o);
                    }
#pragma unroll
                    for (int w = 0; w < UP; ++w) {
                        const int s = s0 + w * nwarp, o = s < NX ? s * G::PSZ : G::SS + (s - NX) * G::PSZ;
#pragma unroll
                        for (int u = 0; u < UE; ++u)
                            if (s < 2 * NX && e0 + 32 * u < R.npull) p[q[u].dst + o] = v[u][w];
                    }
                }
            }
            __syncthreads();
        }

        // ---- all that reads p: F = lam G_j + (lam + mu) sum_{k != j} G_k, and
        // the second derivatives at the own points ---------------------------
        T q[XH][3], pv[XH][3], tau[3];
        if constexpr (ragged) {
#pragma unroll
            for (int x = 0; x < XH; ++x)
#pragma unroll
                for (int c = 0; c < 3; ++c) q[x][c] = pv[x][c] = T(0);
        }
        if (has) {
            auto putf = [&](int x, T a, T b, T c) {
                f1[x * f1s] = a;
                if (x < NX) {
                    f2[x * G::PSa] = b;
                    f3[x * G::PSb] = c;
                }
            };
            res_with_part<NP>(half, [&](auto P) {
                constexpr int A = decltype(P)::value * XH, B = A + XH < NX ? A + XH : NX;
                res_own_p<T, N1, G, A, B>(C, X, line, sgn, row2, row3, q, pv, tau, putf);
            });
        }
        // Halo rows: F2 two rows beyond the tile along x2, F3 along x3.
        for (int u = GRID ? nwarp - 1 - warp : warp; u < NP * (R.nch - R.nch0); u += nwarp) {
            const int ch = R.nch0 + u / NP;
            const bool two = chunks[ch] == 1;
            const ResLine H = lines[ch * kResLinesPerChunk + sub];
            const T *v = p + side * G::SS + H.plo;
            T *f = two ? F2 + side * G::SSa + H.f2 : F3 + side * G::SSb + H.f3;
            const int fs = two ? G::PSa : G::PSb;
            auto put = [&](int x, T G1, T G2, T G3) {
                f[x * fs] = two ? C.lam * G2 + C.lpm * (G1 + G3) : C.lam * G3 + C.lpm * (G1 + G2);
            };
            const ResLineRow<T> h2 = rows(H.info & 15), h3 = rows(9 + (H.info >> 4 & 15));
            res_with_part<NP>(u % NP, [&](auto P) {
                constexpr int A = decltype(P)::value * XH, B = A + XH < NX ? A + XH : NX;
                res_line_grad<T, N1, G, A, B>(X, v, sgn, h2, h3, put);
            });
        }
        __syncthreads();

        // ---- q = A p on the own points, and the dot products -----------------
        double sums[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // p.q, p.p, r.q, q.q, r.r
        if (has) {
            res_with_part<NP>(half, [&](auto P) {
                constexpr int A = decltype(P)::value * XH, B = A + XH < NX ? A + XH : NX;
                res_own_f<T, N1, G, A, B>(X, f1, f1s, f2, f3, sgn, row2, row3, q);
            });
            if (half == 0) {
                // SAT c (tau+ - tau-) on both sides, then P averages the fault node.
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    q[0][j] += C.sat * sgn * (tau[j] - __shfl_xor_sync(0xffffffffu, tau[j], 1));
                    q[0][j] = T(0.5) * (q[0][j] + __shfl_xor_sync(0xffffffffu, q[0][j], 1));
                }
            }
#pragma unroll
            for (int x = 0; x < XH; ++x) {
                T hw = X.hx[x];
#pragma unroll
                for (int P = 1; P < NP; ++P)
                    if (half == P) hw = X.hx[P * XH + x < N1 ? P * XH + x : NX];
                hw *= hw23;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    q[x][c] *= hw;
                    const double qd = (double)q[x][c], pd = own ? (double)pv[x][c] : 0.0;
                    const double rd = (double)r[x][c];
                    sums[0] += pd * qd;
                    sums[1] += pd * pd;
                    sums[2] += rd * qd;
                    sums[3] += qd * qd;
                    sums[4] += rd * rd;
                }
            }
        }
        // Sums of the warp: halving exchanges leave sum `lane >> 2` in each
        // group of four lanes (5 to 7: none); then the CTA's, by warp 0, to
        // every CTA.
        const int sum = lane >> 2, part = lane & 3;
        double h4[4], h2[2], c1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double lo = sums[j], hi = j == 0 ? sums[4] : 0.0;
            h4[j] = ((lane & 16) ? hi : lo) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? lo : hi, 16);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
            h2[j] = ((lane & 8) ? h4[j + 2] : h4[j]) + __shfl_xor_sync(0xffffffffu, (lane & 8) ? h4[j] : h4[j + 2], 8);
        c1 = ((lane & 4) ? h2[1] : h2[0]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? h2[0] : h2[1], 4);
        c1 += __shfl_xor_sync(0xffffffffu, c1, 2);
        c1 += __shfl_xor_sync(0xffffffffu, c1, 1);
        if (part == 0) wred[warp * 8 + sum] = c1;
        __syncthreads();
        if (warp == 0) {
            c1 = wred[part * 8 + sum];
#pragma unroll
            for (int w = 4; w < kResMaxWarps; w += 4) c1 += wred[(part + w) * 8 + sum];  // absent warps hold zero
            c1 += __shfl_xor_sync(0xffffffffu, c1, 2);
            c1 += __shfl_xor_sync(0xffffffffu, c1, 1);
            if constexpr (GRID) {
                if (part == 0) __stcg(team_red + rank * 8 + sum, c1);
            } else if (M > 1) {
                double *to = red + rank * 8 + sum;
#pragma unroll
                for (int w = 0; w < kResMaxTeam; w += 4)
                    if (part + w < M) *map_cluster(to, part + w) = c1;
            } else if (part == 0) {
                red[sum] = c1;
            }
        }
        if (!meet()) return;

        // ---- alpha, beta and the decision, by warp 0 of each CTA --------------
        // The next residual's norm from the same sums, |r - a q|^2 =
        // |r|^2 - 2 a r.q + a^2 q.q: no second exchange. |r|^2 is summed anew
        // each time, so its rounding does not build up; and where FP64 would
        // stop on the difference, or it is small, the new residual is summed
        // too (below; that bound in explicit operations, so that the compiler
        // shares none of them with rr and rounds it alike).
        if (warp == 0) {
            if constexpr (GRID) {
                c1 = 0.0;
                for (int w = part; w < M; w += 4) c1 += __ldcg(team_red + w * 8 + sum);
            } else {
                c1 = red[part * 8 + sum];
#pragma unroll
                for (int w = 4; w < kResMaxTeam; w += 4) c1 += red[(part + w) * 8 + sum];  // ranks beyond M hold zero
            }
            c1 += __shfl_xor_sync(0xffffffffu, c1, 2);
            c1 += __shfl_xor_sync(0xffffffffu, c1, 1);
            const double pq = __shfl_sync(0xffffffffu, c1, 0), pp = __shfl_sync(0xffffffffu, c1, 4),
                         rq = __shfl_sync(0xffffffffu, c1, 8), qq = __shfl_sync(0xffffffffu, c1, 12);
            gamma = __shfl_sync(0xffffffffu, c1, 16);
            double alpha = gamma / pq;
            const bool breakdown = !(pq > 2.220446049250313e-16 * pp);  // zero or negative curvature
            if (breakdown || !isfinite(alpha)) alpha = 0.0;
            const double ad = (double)(T)alpha;
            const double rr = fmax(gamma - 2.0 * ad * rq + ad * ad * qq, 0.0);
            bool sure = true;
            ++iters;
            if (breakdown) {
                if (mixed) flag = 1;  // let the true residual decide
                else status = COL_BREAKDOWN;
            } else if (!isfinite(gamma) || !isfinite(rq) || !isfinite(qq)) {
                status = COL_NONFINITE;
            } else if (mixed) {
                if (rr <= tol * tol || rr <= sp.delta * sp.delta * rr_ref || iters >= itmax) flag = 1;
            } else if (sqrt(rr) <= tol || rr <= 1e-10 * __fma_rn(__dmul_rn(ad, ad), qq, gamma)) {
                sure = false;
            } else if (iters >= itmax) {
                status = COL_MAXITER;
            }
            const bool stop = flag || status != COL_ACTIVE;
            if (!stop) {
                beta = rr / gamma;
            }
            if (lane == 0) {
                step[0] = alpha;
                step[1] = beta;
                step[2] = stop || k + 1 >= kmax ? 1.0 : 0.0;
                step[3] = sure ? 1.0 : 0.0;
            }
        }
        __syncthreads();
        const T at = (T)step[0];
        T b = (T)step[1];
        bool last = step[2] != 0.0;
        if (has) {
#pragma unroll
            for (int x = 0; x < XH; ++x)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    xs[x][c] += at * pv[x][c];
                    r[x][c] -= at * q[x][c];
                }
        }
        if constexpr (sizeof(T) == 8) {
            if (step[3] == 0.0) {
                // The new residual's own norm, exchanged like the sums above in
                // a place that they leave free. FP64 has no true residual to
                // correct a decision, and the norm from the sums is a
                // difference: below about 1e-14 |r|^2 of the old residual it is
                // rounding (a right-hand side within 1e-9 of an eigenvector was
                // called converged after one iteration). Once a column, as a
                // rule.
                constexpr int kOwn = 5;
                double s = 0.0;
                if (has) {
#pragma unroll
                    for (int x = 0; x < XH; ++x)
#pragma unroll
                        for (int c = 0; c < 3; ++c) s += r[x][c] * r[x][c];
                }
                auto warp_sum = [](double v) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    return v;
                };
                s = warp_sum(s);
                if (lane == 0) wred[warp * 8 + kOwn] = s;
                __syncthreads();
                if (warp == 0) {
                    s = warp_sum(lane < kResMaxWarps ? wred[lane * 8 + kOwn] : 0.0);  // absent warps hold zero
                    if constexpr (GRID) {
                        if (lane == 0) __stcg(team_red + rank * 8 + kOwn, s);
                    } else if (lane < M) {
                        *(M > 1 ? map_cluster(red + rank * 8 + kOwn, lane) : red + kOwn) = s;
                    }
                }
                if (!meet()) return;
                if (warp == 0) {
                    s = 0.0;
                    if constexpr (GRID) {
                        for (int w = lane; w < M; w += 32) s += __ldcg(team_red + w * 8 + kOwn);
                    } else if (lane < kResMaxTeam) {
                        s = red[lane * 8 + kOwn];  // ranks beyond M hold zero
                    }
                    const double rr = warp_sum(s);
                    if (sqrt(rr) <= tol) status = COL_CONVERGED;
                    else if (iters >= itmax) status = COL_MAXITER;
                    else beta = rr / gamma;
                    if (lane == 0) {
                        step[1] = beta;
                        if (status != COL_ACTIVE) step[2] = 1.0;
                    }
                }
                __syncthreads();
                b = step[1];
                last = step[2] != 0.0;
            }
        }
        if (last) break;
        if (has) {
#pragma unroll
            for (int x = 0; x < XH; ++x)
#pragma unroll
                for (int c = 0; c < 3; ++c) pv[x][c] = r[x][c] + b * pv[x][c];
            put_p(pv);
        }
    }
    // Leave the state as the streamed iteration does: p is the last
    // iteration's direction, beta the next one's factor.
    if (own) {
#pragma unroll
        for (int x = 0; x < XH; ++x)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (!live(x)) continue;
                const long long g = g0 + c * (long long)cstr + x * gstep;
                x_[g] = xs[x][c];
                p_[g] = mine[x * G::PSZ + c * G::CS];
                r_[g] = r[x][c];
            }
    }
    if (rank == 0 && tid == 0) {
        st.iters[slot] = iters;
        st.beta[slot] = beta;
        st.gamma[slot] = gamma;
        if (mixed) st.flag[slot] = (int8_t)flag;
        if (status != COL_ACTIVE) st.status[slot] = (int8_t)status;
    }
    }
}

}  // namespace eqd
