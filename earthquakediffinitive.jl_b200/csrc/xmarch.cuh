// x1 march: the FP32 CG apply q = -H P (D + SAT) p of the streamed iteration,
// for vectors stored x2-fastest.
//
// The plane marches (plane_march.cuh, ring_march.cuh) step along x3 over
// vectors stored x1-fastest: a thread has one point, reads its x1 neighbours
// from shared memory with per-lane rows, and pays about 520 instructions a
// point (900 GB/s at h = 20 m). Here vectors are stored
//   v[col][side][comp][x][i3][n2p],  x = 0 at the fault on both sides
// (a column that 32-bit byte offsets reach: x_offsets_fit),
// x2 line i2 at 3 + i2 of a row padded to a multiple of 4 (so that tiles, which
// start at i2 = 1 mod 4, have their halo on a 16-byte boundary), and a CTA owns
// a tile of 16 x 8 (x2, x3) lines of both sides and steps outwards from the
// fault:
//   * a thread has one line; x1 derivatives come from 7-deep register windows
//     with one row for the whole CTA (no x1 loads, no divergence at closures);
//   * x2 and x3 neighbours come from the step's plane in shared memory, by
//     rows that depend on the line only and stay in registers (interior and
//     closure lines run the same code);
//   * planes (tile and four halo lines around it, both sides, three
//     components) arrive by one tiled bulk-tensor copy each, three ahead of
//     use; lines beyond the domain arrive as zeros;
//   * F_2 and F_3 go through shared memory (one barrier a step); the threads
//     also march the F of the two halo lines that each neighbour direction
//     needs;
//   * the two sides of a line sit in adjacent lanes: SAT and P by shuffle;
//   * seven steps are unrolled, the depth of the windows and of every ring, so
//     that all ring places are immediate offsets (with run-time places 430
//     instructions were issued a line and step, 300 of them addresses and
//     moves).
// Operator and factorisation as in resident_cg.cuh.
//
// What bounds it: instruction issue (0.58 of the schedulers' slots, 256
// instructions a line and step). Measured at h = 20 m, 48 columns: 201 us, the
// plane march 360; 320-thread tiles of 16 x 10 lines (96 registers, spilling)
// 309. 96 columns' solves there 293 ms (458 with the plane march and its
// vector kernels), ten columns at h = 25 m 193 ms (370).
//
// Dot products p.q and q.q are summed per (column, tile) in a fixed order.
#pragma once
#include <cuda.h>

#include "resident_cg.cuh"
#include "xmarch_plan.h"

namespace eqd {

constexpr int kXT2 = 16, kXT3 = 8;                      // own lines of a CTA
constexpr int kXR2 = kXT2 + 8, kXR3 = kXT3 + 8 + 2;     // with four halo lines around them (two rows more: see kXSS below)
constexpr int kXPSZ = kXR2 * kXR3, kXSS = 3 * kXPSZ;    // component and side strides of a plane
constexpr int kXRing = 7;                               // planes and F buffers; planes c .. c + 3 are in use
constexpr int kXPlane = 2 * kXSS;                       // elements of a plane
constexpr int kXThreads = 2 * kXT2 * kXT3;
constexpr int kXR2a = kXT2 + 4;                         // row of F_2: two halo lines along x2
constexpr int kXF2 = kXR2a * kXT3 + 16, kXF3 = kXT2 * (kXT3 + 4) + 16;  // one side's F_2 and F_3
constexpr int kXF = 2 * (kXF2 + kXF3);                  // one step's F: both sides of F_2, then of F_3
static_assert(kXSS % 32 == 16 && kXF2 % 32 == 16 && kXF3 % 32 == 16, "the two sides of a warp's lines fall on distinct banks");
static_assert(kXPlane * 4 % 128 == 0, "a plane starts on a 128-byte boundary");
constexpr int kXSmemRows = 128 + kXRing * kXPlane * 4;  // byte offset of the x1 rows
constexpr int xmarch_smem(int n1) { return kXSmemRows + n1 * 16 * 4 + kXRing * kXF * 4; }

struct XGeom {
    int n1, n2, n3, n2p;
    long long colstride;
    int nt2, nt3;             // tiles
    const int *b2, *b3;       // their first lines, and the end
    const float *rows;        // x1 rows, 16 floats: D1 at -3..3, mu D2 at -3..3, -hvol times the weight
    const float *tab;         // fill_res_tables rows of x2, then x3
    const int *off;
};

struct XCoef {
    float lam, lpm, mu, mu2, sat;
    float a, b;               // interior D1 of x1
    float s0, s1, s2;         // interior mu D2 of x1
    float dlo[4];
};

__device__ __forceinline__ void tma_plane(void *dst, const CUtensorMap *map, int x2, int x3, int x, int col,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
        "[%7];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x2), "r"(x3), "r"(x), "r"(0), "r"(col), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ float x_dot4(const float (&c)[4], float t0, float t1, float t2, float t3) {
    return c[0] * t0 + c[1] * t1 + c[2] * t2 + c[3] * t3;
}

__device__ __forceinline__ int x_class(int i, int n) { return i < 4 ? i : (i >= n - 4 ? 5 + (n - 1 - i) : 4); }

// Shared memory at a thread's address plus a constant number of elements: the
// constant goes into the instruction (through pointers the compiler formed
// most of these addresses again at every use).
template <int AT>
__device__ __forceinline__ float x_ld(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(AT * 4));
    return v;
}
template <int AT>
__device__ __forceinline__ void x_st(unsigned a, float v) {
    asm volatile("st.shared.f32 [%0+%1], %2;" ::"r"(a), "n"(AT * 4), "f"(v) : "memory");
}

// An x1 row (the same for every thread).
__device__ __forceinline__ void x_row16(unsigned a, float (&r)[16]) {
#pragma unroll
    for (int k = 0; k < 16; k += 4)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(r[k]), "=f"(r[k + 1]), "=f"(r[k + 2]), "=f"(r[k + 3])
                     : "r"(a + 4 * k));
}

__device__ __forceinline__ bool x_wait(unsigned bar, unsigned parity, unsigned *err) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    return mbar_wait_bounded(reinterpret_cast<uint64_t *>(__cvta_shared_to_generic(bar)), parity, err);
}

// Row of an x1 operator on a window ring: entry o of the row meets plane
// centre + o, which sits at ring place (C0 + o) mod 7.
template <int C0>
__device__ __forceinline__ float x_dot7(const float (&row)[16], int at, const float (&w)[kXRing]) {
    float s = row[at] * w[(C0 + 4) % 7];
#pragma unroll
    for (int k = 1; k < 7; ++k) s += row[at + k] * w[(C0 + k + 4) % 7];
    return s;
}
template <int C0>
__device__ __forceinline__ float x_first(const XCoef &C, const float (&w)[kXRing]) {
    return C.a * (w[(C0 + 1) % 7] - w[(C0 + 6) % 7]) + C.b * (w[(C0 + 2) % 7] - w[(C0 + 5) % 7]);
}
template <int C0>
__device__ __forceinline__ float x_second(const XCoef &C, const float (&w)[kXRing]) {
    return C.s0 * w[C0] + C.s1 * (w[(C0 + 6) % 7] + w[(C0 + 1) % 7]) + C.s2 * (w[(C0 + 5) % 7] + w[(C0 + 2) % 7]);
}

// What a thread keeps during the march; places are shared-memory addresses in
// ring place 0.
struct XThread {
    unsigned o;                  // own line; component stride kXPSZ
    unsigned oa2, ob2, oa3, ob3; // outer places of the x2 and x3 rows (the inner ones are the neighbours)
    float c2[4], c3[4], s2[5], s3[5];  // D1 and mu D2
    unsigned f2, fa2, fb2;       // own place in F_2, and the outer ones of its row
    unsigned f3, fa3, fb3;       // the same in F_3
    unsigned h, u2[4], u3[4];    // halo line, and the places of its D1 rows (in v_2, in v_3)
    float d2[4], d3[4];
    unsigned hf;                 // and its F
    float hc2, hc3;              // weights of G_2 and G_3 in it
    float sgn, hw23;
    bool own, hal, first;        // carries unknowns; has a halo line; thread 0
    unsigned q;                  // own line in the column: component 1, x = 0 (bytes)
    unsigned bar, rows;          // the mbarriers, the x1 rows
};

struct XState {
    float v1[kXRing], v2[kXRing], v3[kXRing], F1[kXRing], w1[kXRing], hv[kXRing];
    double acc0, acc1;
};

// Step s = 7 t + J: plane s arrives (ring place J); F and components 2, 3 of
// c = s - 3; component 1 of e = s - 6 (its D1_1 F_1 reads F_1 of e - 3 .. e + 3).
// False when a wait gave up.
template <int J, typename ISSUE>
__device__ __forceinline__ bool x_step(const XGeom &g, const XCoef &C, const XThread &t, XState &S, int s, unsigned parity,
                                       char *qcol, unsigned *err, ISSUE issue) {
    constexpr int PC = (J + 4) % 7, PE = (J + 1) % 7;  // ring places of c and e
    const int n1 = g.n1, c = s - 3, e = s - 6;
    bool ok = true;
    S.v1[J] = S.v2[J] = S.v3[J] = S.hv[J] = 0.f;
    if (s < n1) {
        ok = x_wait(t.bar + 8 * J, parity, err);
        constexpr int P = J * kXPlane;
        S.v1[J] = x_ld<P>(t.o);
        S.v2[J] = x_ld<P + kXPSZ>(t.o);
        S.v3[J] = x_ld<P + 2 * kXPSZ>(t.o);
        S.hv[J] = x_ld<P>(t.h);
    }
    float w1 = 0.f, w2 = 0.f, w3 = 0.f;
    S.F1[PC] = 0.f;
    if (c >= 0 && c < n1) {
        float G1, H1;
        if (c >= 4 && c < n1 - 4) {
            G1 = x_first<PC>(C, S.v1);
            H1 = x_first<PC>(C, S.hv);
            w1 = x_second<PC>(C, S.v1);
            w2 = x_second<PC>(C, S.v2);
            w3 = x_second<PC>(C, S.v3);
        } else {
            float row[16];
            x_row16(t.rows + 64 * c, row);
            G1 = x_dot7<PC>(row, 0, S.v1);
            H1 = x_dot7<PC>(row, 0, S.hv);
            w1 = x_dot7<PC>(row, 7, S.v1);
            w2 = x_dot7<PC>(row, 7, S.v2);
            w3 = x_dot7<PC>(row, 7, S.v3);
        }
        G1 *= t.sgn;
        H1 *= t.sgn;
        float G2, G3, d2 = 0.f, d3 = 0.f;
        constexpr int P = PC * kXPlane;
        // x2 and x3 rows of component j (ring offset AT) at the own line.
#define EQD_XTAPS(AT, own)                                                                                             \
    const float a2 = x_ld<AT>(t.oa2), m2 = x_ld<(AT) - 1>(t.o), p2 = x_ld<(AT) + 1>(t.o), b2 = x_ld<AT>(t.ob2);        \
    const float a3 = x_ld<AT>(t.oa3), m3 = x_ld<(AT) - kXR2>(t.o), p3 = x_ld<(AT) + kXR2>(t.o), b3 = x_ld<AT>(t.ob3);  \
    const float x2 = t.s2[0] * a2 + t.s2[1] * m2 + t.s2[2] * own + t.s2[3] * p2 + t.s2[4] * b2;                        \
    const float x3 = t.s3[0] * a3 + t.s3[1] * m3 + t.s3[2] * own + t.s3[3] * p3 + t.s3[4] * b3;
        {
            EQD_XTAPS(P, S.v1[PC])
            w1 = 2.f * w1 + x2 + x3;
            if (c == 0) {
                d2 = x_dot4(t.c2, a2, m2, p2, b2);
                d3 = x_dot4(t.c3, a3, m3, p3, b3);
            }
        }
        {
            EQD_XTAPS(P + kXPSZ, S.v2[PC])
            w2 += 2.f * x2 + x3;
            G2 = x_dot4(t.c2, a2, m2, p2, b2);
        }
        {
            EQD_XTAPS(P + 2 * kXPSZ, S.v3[PC])
            w3 += x2 + 2.f * x3;
            G3 = x_dot4(t.c3, a3, m3, p3, b3);
        }
#undef EQD_XTAPS
        S.F1[PC] = C.lam * G1 + C.lpm * (G2 + G3);
        x_st<J * kXF>(t.f2, C.lam * G2 + C.lpm * (G1 + G3));
        x_st<J * kXF>(t.f3, C.lam * G3 + C.lpm * (G1 + G2));
        if (t.hal) {
            const float g2 = x_dot4(t.d2, x_ld<P>(t.u2[0]), x_ld<P>(t.u2[1]), x_ld<P>(t.u2[2]), x_ld<P>(t.u2[3]));
            const float g3 = x_dot4(t.d3, x_ld<P>(t.u3[0]), x_ld<P>(t.u3[1]), x_ld<P>(t.u3[2]), x_ld<P>(t.u3[3]));
            x_st<J * kXF>(t.hf, C.lpm * H1 + t.hc2 * g2 + t.hc3 * g3);
        }
        if (c == 0) {
            // SAT c (tau+ - tau-) on both sides; traction on the fixed +x1 axis.
            float h[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                h[0] += C.dlo[k] * S.v1[(PC + k) % 7];
                h[1] += C.dlo[k] * S.v2[(PC + k) % 7];
                h[2] += C.dlo[k] * S.v3[(PC + k) % 7];
            }
            const float t1 = C.lam * (G1 + G2 + G3) + C.mu2 * (t.sgn * h[0]);
            const float t2 = C.mu * (d2 + t.sgn * h[1]), t3 = C.mu * (d3 + t.sgn * h[2]);
            w1 += C.sat * t.sgn * (t1 - __shfl_xor_sync(0xffffffffu, t1, 1));
            w2 += C.sat * t.sgn * (t2 - __shfl_xor_sync(0xffffffffu, t2, 1));
            w3 += C.sat * t.sgn * (t3 - __shfl_xor_sync(0xffffffffu, t3, 1));
        }
    }
    S.w1[PC] = w1;
    if (__syncthreads_or(!ok)) return false;
    // Every thread has read plane c for the last time: its ring place is free.
    if (t.first && c >= 0 && c + kXRing < n1) issue(c + kXRing, PC);
    const unsigned qx = 4u * (unsigned)(g.n3 * g.n2p), qc = qx * (unsigned)n1;  // bytes from x to x, and component to component
    if (c >= 0 && c < n1 - 1) {
        constexpr int P = J * kXF;
        w2 += x_dot4(t.c2, x_ld<P>(t.fa2), x_ld<P - 1>(t.f2), x_ld<P + 1>(t.f2), x_ld<P>(t.fb2));
        w3 += x_dot4(t.c3, x_ld<P>(t.fa3), x_ld<P - kXT2>(t.f3), x_ld<P + kXT2>(t.f3), x_ld<P>(t.fb3));
        if (c == 0) {
            w2 = 0.5f * (w2 + __shfl_xor_sync(0xffffffffu, w2, 1));
            w3 = 0.5f * (w3 + __shfl_xor_sync(0xffffffffu, w3, 1));
        }
        const float hw = x_ld<14>(t.rows + 64 * c) * t.hw23, q2 = hw * w2, q3 = hw * w3;
        const unsigned at = t.q + (unsigned)c * qx + qc;
        if (t.own) {
            *reinterpret_cast<float *>(qcol + at) = q2;
            *reinterpret_cast<float *>(qcol + at + qc) = q3;
        }
        const double p2 = t.own ? (double)S.v2[PC] : 0.0, p3 = t.own ? (double)S.v3[PC] : 0.0;
        S.acc0 = fma(p2, (double)q2, S.acc0);
        S.acc1 = fma((double)q2, (double)q2, S.acc1);
        S.acc0 = fma(p3, (double)q3, S.acc0);
        S.acc1 = fma((double)q3, (double)q3, S.acc1);
    }
    if (e >= 0 && e < n1 - 1) {
        float E;
        if (e >= 4 && e < n1 - 4) {
            E = x_first<PE>(C, S.F1);
        } else {
            float row[16];
            x_row16(t.rows + 64 * e, row);
            E = x_dot7<PE>(row, 0, S.F1);
        }
        float w = S.w1[PE] + t.sgn * E;
        if (e == 0) w = 0.5f * (w + __shfl_xor_sync(0xffffffffu, w, 1));
        const float q1 = x_ld<14>(t.rows + 64 * e) * t.hw23 * w;
        if (t.own) *reinterpret_cast<float *>(qcol + (t.q + (unsigned)e * qx)) = q1;
        const double p1 = t.own ? (double)S.v1[PE] : 0.0;
        S.acc0 = fma(p1, (double)q1, S.acc0);
        S.acc1 = fma((double)q1, (double)q1, S.acc1);
    }
    return true;
}

__global__ void __launch_bounds__(kXThreads, 2)
xmarch_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ XGeom g,
              const __grid_constant__ XCoef C, float *__restrict__ q, const int8_t *__restrict__ status,
              double *__restrict__ partials, int col0, unsigned *__restrict__ err) {
    const int ntiles = g.nt2 * g.nt3;
    const int col = blockIdx.x / ntiles, tile = blockIdx.x % ntiles;  // columns of this launch start at col0 of the map
    if (status && status[col] != COL_ACTIVE) return;
    const int n1 = g.n1, n2 = g.n2, n3 = g.n3;
    const int a2 = g.b2[tile % g.nt2], e2 = g.b2[tile % g.nt2 + 1], a3 = g.b3[tile / g.nt2], e3 = g.b3[tile / g.nt2 + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem_raw);
    float *ring = reinterpret_cast<float *>(smem_raw + 128);
    float *rows = reinterpret_cast<float *>(smem_raw + kXSmemRows);
    float *F = rows + n1 * 16;
    __shared__ double red[32];

    for (int i = tid; i < n1 * 16; i += kXThreads) rows[i] = g.rows[i];
    for (int i = tid; i < kXRing * kXF; i += kXThreads) F[i] = 0.f;
    if (tid == 0) {
        for (int k = 0; k < kXRing; ++k) mbar_init(&mbar[k], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int s, int place) {
        mbar_arrive_expect_tx(&mbar[place], kXPlane * 4);
        tma_plane(ring + place * kXPlane, &map, a2 - 4 + kXLead, a3 - 4, s, col0 + col, &mbar[place]);
    };
    if (tid == 0)
        for (int s = 0; s < min(kXRing, n1); ++s) issue(s, s);

    // Own line: warp w has the tile's x3 row w, its 16 lines along x2, both sides.
    XThread t;
    const int side = lane & 1, k2 = lane >> 1, k3 = warp, i2 = a2 + k2, i3 = a3 + k3;
    t.sgn = side ? 1.f : -1.f;
    t.own = i2 < e2 && i3 < e3;
    const unsigned ring0 = smem_u32(ring), F0 = smem_u32(F);
    t.o = ring0 + 4 * (side * kXSS + (k3 + 4) * kXR2 + k2 + 4);
    const int cls2 = t.own ? x_class(i2, n2) : 4, cls3 = 9 + (t.own ? x_class(i3, n3) : 4);
    const float *tab2 = g.tab + cls2 * kResRow, *tab3 = g.tab + cls3 * kResRow;
    const int *of2 = g.off + cls2 * 4, *of3 = g.off + cls3 * 4;
    t.oa2 = t.o + 4 * of2[0];
    t.ob2 = t.o + 4 * of2[3];
    t.oa3 = t.o + 4 * kXR2 * of3[0];
    t.ob3 = t.o + 4 * kXR2 * of3[3];
    t.f2 = F0 + 4 * (side * kXF2 + k3 * kXR2a + k2 + 2);
    t.fa2 = t.f2 + 4 * of2[0];
    t.fb2 = t.f2 + 4 * of2[3];
    t.f3 = F0 + 4 * (2 * kXF2 + side * kXF3 + (k3 + 2) * kXT2 + k2);
    t.fa3 = t.f3 + 4 * kXT2 * of3[0];
    t.fb3 = t.f3 + 4 * kXT2 * of3[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        t.c2[k] = tab2[k];
        t.c3[k] = tab3[k];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        t.s2[k] = tab2[4 + k];
        t.s3[k] = tab3[4 + k];
    }
    t.hw23 = t.own ? tab2[9] * tab3[9] : 0.f;
    if (!t.own) {  // a narrower tile's idle threads: out of the way of its halo lines, in the padding of F_3's side 0
        t.f2 = t.f3 = F0 + 4 * (2 * kXF2 + kXF3 - 16);
        t.fa2 = t.fb2 = t.fa3 = t.fb3 = t.f2;
    }
    t.first = tid == 0;
    t.bar = smem_u32(mbar);
    t.rows = smem_u32(rows);
    t.q = 4u * (unsigned)(side * 3 * n1 * n3 * g.n2p + i3 * g.n2p + i2 + kXLead);

    // Halo line: threads 0 .. 127 those of F_3 (four rows of 16 lines), the next
    // 8 kXT3 those of F_2 (four lines of each row).
    int h2 = 0, h3 = 0, hf = 0;
    bool two = false;
    t.hal = false;
    if (tid < 128) {
        h3 = warp < 2 ? a3 - 2 + warp : e3 + warp - 2;  // two rows before the tile, two after
        h2 = i2;
        t.hal = h2 < e2 && h3 >= 0 && h3 < n3;
        hf = 2 * kXF2 + side * kXF3 + (h3 - a3 + 2) * kXT2 + k2;
    } else if (tid < 128 + 8 * kXT3) {
        const int k = (tid - 128) >> 1, at = k & 3;
        h2 = at < 2 ? a2 - 2 + at : e2 + at - 2;
        h3 = a3 + (k >> 2);
        t.hal = two = h3 < e3 && h2 >= 0 && h2 < n2;
        hf = side * kXF2 + (h3 - a3) * kXR2a + h2 - a2 + 2;
    }
    t.h = ring0 + 4 * (t.hal ? side * kXSS + (h3 - a3 + 4) * kXR2 + h2 - a2 + 4 : 0);
    t.hf = F0 + 4 * (t.hal ? hf : 0);
    const int hc2 = t.hal ? x_class(h2, n2) : 4, hc3 = 9 + (t.hal ? x_class(h3, n3) : 4);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        t.d2[k] = g.tab[hc2 * kResRow + k];
        t.d3[k] = g.tab[hc3 * kResRow + k];
        t.u2[k] = t.h + 4 * (kXPSZ + (t.hal ? g.off[hc2 * 4 + k] : 0));
        t.u3[k] = t.h + 4 * (2 * kXPSZ + (t.hal ? g.off[hc3 * 4 + k] * kXR2 : 0));
    }
    t.hc2 = two ? C.lam : C.lpm;
    t.hc3 = two ? C.lpm : C.lam;

    XState S;
#pragma unroll
    for (int k = 0; k < kXRing; ++k) S.v1[k] = S.v2[k] = S.v3[k] = S.F1[k] = S.w1[k] = S.hv[k] = 0.f;
    S.acc0 = S.acc1 = 0.0;
    char *qcol = reinterpret_cast<char *>(q + (long long)col * g.colstride);
    const int last = n1 + 5;  // e reaches n1 - 2
    bool ok = true;
    int s = 0;
    for (unsigned trip = 0; ok && s < last; ++trip) {
        const unsigned par = trip & 1u;
#define EQD_XSTEP(J)                                                                       \
    if (ok && s < last) {                                                                  \
        ok = x_step<J>(g, C, t, S, s, par, qcol, err, issue);                                 \
        s += ok;                                                                           \
    }
        EQD_XSTEP(0) EQD_XSTEP(1) EQD_XSTEP(2) EQD_XSTEP(3) EQD_XSTEP(4) EQD_XSTEP(5) EQD_XSTEP(6)
#undef EQD_XSTEP
    }
    if (!ok) {
        // A wait gave up at step s (recorded in *err): planes s .. min(s + 3, n1 - 1)
        // are under way (plane c + 7 = s + 4 is issued after step s); no copy may
        // land after the CTA has left.
        if (tid == 0)
            for (int p = s; p < min(max(s + 4, kXRing), n1); ++p)
                mbar_wait_bounded(&mbar[p % kXRing], (unsigned)(p / kXRing) & 1u, err);
        __syncthreads();
        return;
    }
    const double t0 = block_sum(S.acc0, red);
    __syncthreads();
    const double t1 = block_sum(S.acc1, red);
    if (tid == 0 && partials) {
        double *pp = partials + ((long long)col * ntiles + tile) * 2;
        pp[0] = t0;
        pp[1] = t1;
    }
}

// Between the two layouts, for the flagged (or masked) columns: an item is one
// column's side and component, x3 plane and 32 lines along x2, transposed
// through shared memory so that both sides move whole sectors.
struct XLayout {
    int n1, n2, n3, n2p, PS;
    long long cold, cnew;   // column strides of the x1-fastest and the x2-fastest vectors
};

// FOLD: x += d, d = 0 (x FP64, x1-fastest; d x2-fastest). Else: r = src (src
// x1-fastest, r in d, x2-fastest) and p += the change of r, so that p = r +
// beta p holds for the new r (a column that enters has r = p = 0: p = r). src
// is q's memory, column after column at the x1-fastest stride (which is no
// longer, x_column): zeroed once read, so that q's padding, which the step
// kernel reads, is zero again. The rest of q the next apply writes.
// The blocks share out the items of the flagged columns, of which there are
// usually none or a few: one column then has the whole chip (a few blocks to
// each column took 100 to 170 us whenever one was flagged, of 400 an iteration
// of 48 columns at h = 20 m).
constexpr int kXLayoutBlocks = 592;  // four an SM
template <bool FOLD>
__global__ void __launch_bounds__(256) xlayout_kernel(XLayout g, double *__restrict__ x, float *__restrict__ d,
                                                      float *__restrict__ src, float *__restrict__ p,
                                                      const int8_t *__restrict__ status,
                                                      const int8_t *__restrict__ flag, int ncols) {
    __shared__ float t[32][EQD_MAX_N1 + 1];
    const int nb = (g.n2 + 31) / 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = 6 * g.n3 * nb;  // items of a column: side and component, x3 plane, 32 lines along x2
    const long long xs = (long long)g.n3 * g.n2p;
    int k0 = blockIdx.x;  // this block's next item, counted from the current flagged column's first
    for (int cb = 0; cb < ncols; cb += 32) {
        const bool f = cb + lane < ncols && status[cb + lane] == COL_ACTIVE && flag[cb + lane];
        for (unsigned m32 = __ballot_sync(0xffffffffu, f); m32; m32 &= m32 - 1) {
            const int col = cb + __ffs(m32) - 1;
            for (; k0 < per; k0 += gridDim.x) {
                const int b = k0 % nb, i3 = k0 / nb % g.n3, sc = k0 / nb / g.n3, side = sc / 3;
                const int i2b = b * 32, m = min(32, g.n2 - i2b);
                const long long at = col * g.cnew + ((long long)sc * g.n1 * g.n3 + i3) * g.n2p + i2b + kXLead;
                const long long po = col * g.cold + ((long long)sc * g.n3 + i3) * g.PS + (long long)i2b * g.n1;
                float *dn = d + at;
                if (FOLD) {
                    for (int xx = warp; xx < g.n1; xx += 8)
                        if (lane < m) {
                            t[lane][side ? xx : g.n1 - 1 - xx] = dn[xx * xs + lane];
                            dn[xx * xs + lane] = 0.f;
                        }
                    __syncthreads();
                    for (int i = threadIdx.x; i < m * g.n1; i += 256) x[po + i] += (double)t[i / g.n1][i % g.n1];
                } else {
                    for (int i = threadIdx.x; i < m * g.n1; i += 256) t[i / g.n1][i % g.n1] = src[po + i];
                    __syncthreads();
                    for (int i = threadIdx.x; i < m * g.n1; i += 256) src[po + i] = 0.f;  // (apart: the loads stay in flight)
                    for (int xx = warp; xx < g.n1; xx += 8)
                        if (lane < m) {
                            const float v = t[lane][side ? xx : g.n1 - 1 - xx];
                            p[at + xx * xs + lane] += v - dn[xx * xs + lane];
                            dn[xx * xs + lane] = v;
                        }
                }
                __syncthreads();
            }
            k0 -= per;
        }
    }
}

// Reference order (FP64) <-> x2-fastest vectors (FP32); for the operator hook.
template <bool TO>
__global__ void xref_kernel(XLayout g, double *__restrict__ ref, float *__restrict__ v, int ncols) {
    const long long N = (long long)g.n1 * g.n2 * g.n3, ntot = 6 * N;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= ntot * ncols) return;
    const long long col = gid / ntot, r = gid % ntot, sc = r / N, pt = r % N;
    const int i1 = (int)(pt % g.n1), i2 = (int)(pt / g.n1 % g.n2), i3 = (int)(pt / g.n1 / g.n2);
    const int x = sc >= 3 ? i1 : g.n1 - 1 - i1;
    float *at = v + col * g.cnew + ((sc * g.n1 + x) * g.n3 + i3) * g.n2p + i2 + kXLead;
    if (TO) *at = (float)ref[gid];
    else ref[gid] = (double)*at;
}

}  // namespace eqd
