// Host-side plan of the resident CG (resident_cg.cuh): how one column is
// split over the CTAs of a cluster, and the tables the kernel reads.
//
// A "line" is the set of x1 points of one (x2, x3) node, both sides. The
// lines that carry unknowns are the ones off the far-field ring
// (1 <= i2 <= n2-2, 1 <= i3 <= n3-2); they are split into Mt2 x Mt3
// rectangular tiles, one per CTA. x1 is stored from the fault outwards on
// both sides (x = 0 at the fault, x = n1-1 at the far field), so both sides
// run the same stencil with the sign of D1_1 flipped on the minus side.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "ops_tables.h"

#ifdef __CUDACC__
#define EQD_HD __host__ __device__
#else
#define EQD_HD
#endif

namespace eqd {

constexpr int kResMaxTeam = 16;        // CTAs of a cluster
constexpr int kResMaxGridTeam = 100;   // CTAs of a team that meets through global memory
constexpr int kResMaxWarps = 16;       // of a CTA: one per chunk of own lines and part of the lines
constexpr int kResLinesPerChunk = 16;  // a warp holds 16 lines x 2 sides, the sides of a line in adjacent lanes
constexpr int kResRow = 12;            // elements of a table row (fill_res_tables)
constexpr size_t kResSmemMax = 232448; // 227 KB, the most a CTA of sm_100 may use

// The planes a kernel instance is compiled for: tiles of at most T2 x T3 own
// lines, n1 = N1, elements of EB bytes. Every stride is a constant, so every
// neighbour is an immediate offset (with run-time strides more than half of
// the issued instructions were address arithmetic). Sides are offset so that
// the sixteen lines of a warp (two rows of eight) and their other sides fall
// on distinct banks.
template <int EB, int N1, int T2, int T3>
struct ResGeo {
    static constexpr int n1 = N1;
    static constexpr int NX = N1 - 1;                       // p and F2, F3 need no far-field plane
    static constexpr int R2 = T2 + 8, R3 = T3 + 8;
    static constexpr int lanes = EB == 8 ? 16 : 32;         // elements per bank row
    static constexpr int pad(int n, int want) { return n + ((want - n % lanes) + lanes) % lanes; }
    static constexpr int PSZ = R2 * R3, SS = pad(NX * PSZ, 8), CS = 2 * SS;
    static constexpr int R2a = T2 + 8, PSa = R2a * T3, SSa = pad(NX * PSa, 8);       // F2: two halo rows along x2
    static constexpr int R2b = T2, PSb = R2b * (T3 + 4), SSb = pad(NX * PSb, EB == 8 ? 8 : 16);  // F3: along x3
    static constexpr int nch0 = (T2 * T3 + kResLinesPerChunk - 1) / kResLinesPerChunk;
    static constexpr int nch = nch0 + (4 * T3 + kResLinesPerChunk - 1) / kResLinesPerChunk +
                               (4 * T2 + kResLinesPerChunk - 1) / kResLinesPerChunk;
    // Shared-memory layout, bytes; the push table follows.
    static constexpr int align(int o) { return (o + 15) / 16 * 16; }
    static constexpr int oF1 = align(3 * CS * EB);
    static constexpr int oF2 = align(oF1 + N1 * nch0 * 32 * EB);
    static constexpr int oF3 = align(oF2 + 2 * SSa * EB);
    static constexpr int oTab = align(oF3 + 2 * SSb * EB);
    static constexpr int oOff = align(oTab + 18 * kResRow * EB);
    static constexpr int oRed = align(oOff + 18 * 4 * 4);
    static constexpr int oLine = align(oRed + (kResMaxTeam + kResMaxWarps + 1) * 8 * 8);
    static constexpr int oChunk = align(oLine + nch * kResLinesPerChunk * 16);
    static constexpr int oPush = align(oChunk + nch * 4);
};

// The same numbers for the plan builder.
struct ResStrides {
    int T2, T3, R2, R2a, R2b, CS, nch0, oPush;
};

template <int EB, int N1, int T2, int T3>
inline ResStrides res_strides() {
    using G = ResGeo<EB, N1, T2, T3>;
    return ResStrides{T2, T3, G::R2, G::R2a, G::R2b, G::CS, G::nch0, G::oPush};
}

// One line of a chunk: offsets of the line in the p, F2 and F3 planes, and
// info = x2 row class | x3 row class << 4 | valid << 8. Row classes: 0..3
// lower closure rows, 4 interior, 5..8 upper closure rows n-1..n-4.
struct alignas(16) ResLine {
    int plo, f2, f3, info;
};

// What one CTA of the team owns (tables are concatenated over the ranks).
struct ResRank {
    int nch, nch0;        // chunks; the first nch0 hold this CTA's own lines
    int chunk0;
    int push0;            // first row of its own lines in the push table
    int pull0, npull;     // its halo in the pull table
};

// One halo line of one component: where it is in the team's copy of p (a rank's
// part is 3 CS long), and in this CTA's p.
struct alignas(8) ResPull {
    int src, dst;
};

// Chunk types: 0 own lines, 1 F2 halo rows, 2 F3 halo rows.
struct ResDims {
    int n3, PS;
    long long colstride;
    int M, Mt2, Mt3;
    int nch0max, nhalomax;    // a CTA has a warp per chunk of own lines and part of the lines
    int npush;                // places a line's p may have to be pushed to
    int smem;                 // bytes
};

struct ResPlan {
    ResDims d{};
    std::vector<ResRank> ranks;
    std::vector<int> chunks;
    std::vector<ResLine> lines;   // 16 per chunk
    std::vector<int> gofs;        // i3 * PS + i2 * n1 of the line
    // npush words per own line (16 per chunk): rank << 28 | components << 24 | offset of the line in that rank's
    // p; -1: none. A line's new p goes to every CTA that has it in its halo.
    std::vector<int> push;
    std::vector<ResPull> pull;    // the same, as the reader sees it
    double cost = 0;              // warps' work of one iteration over the team
};

inline int res_class(int i, int n) { return i < 4 ? i : (i >= n - 4 ? 5 + (n - 1 - i) : 4); }

// Tile bounds along one axis: `parts` tiles over the rows 1 .. n-2. With more
// than one tile the first and the last hold the three closure rows that carry
// unknowns (a tile sees 2 rows of F and 4 rows of p beyond its own), and no
// tile starts at row 5 or ends before row n-5: its second F halo row would be
// the closure row that reaches five rows back.
inline bool res_split(int n, int parts, std::vector<int> &b) {
    const int m = n - 2;
    if (parts == 1) {
        b = {1, n - 1};
        return m >= 1;
    }
    int best = 1 << 30;
    for (int f = 3; f < m; ++f) {
        for (int l = 3; f + l <= m; ++l) {
            const int rest = m - f - l, k = parts - 2;
            if (k == 0 ? rest != 0 : rest < k) continue;
            const int mid = k ? (rest + k - 1) / k : 0;
            const int mx = std::max({f, l, mid});
            // the widest tile decides; then middle tiles, which have halos on both sides, prefer fewer rows
            const int score = mx * 64 + mid;
            if (score >= best) continue;
            std::vector<int> c = {1, 1 + f};
            for (int q = 1; q < k; ++q) c.push_back(1 + f + (int)((long long)q * rest / k));
            if (k) c.push_back(1 + f + rest);
            c.push_back(n - 1);
            if (std::find(c.begin(), c.end(), 5) != c.end() || std::find(c.begin(), c.end(), n - 5) != c.end()) continue;
            best = score;
            b = c;
        }
    }
    return best < (1 << 30);
}

// The plan of n1 x n2 x n3 nodes on a team of M = Mt2 x Mt3 CTAs; false if a
// tile does not fit the planes of `s`. `pull`: the halo is read by its owner
// (a rank beyond 15 does not fit a push word).
inline bool make_res_plan(int n1, int n2, int n3, int PS, int Mt2, int Mt3, const ResStrides &s, ResPlan &out,
                          bool pull = false) {
    std::vector<int> b2, b3;
    if (!res_split(n2, Mt2, b2) || !res_split(n3, Mt3, b3)) return false;
    for (int k = 0; k < Mt2; ++k)
        if (b2[k + 1] - b2[k] > s.T2) return false;
    for (int k = 0; k < Mt3; ++k)
        if (b3[k + 1] - b3[k] > s.T3) return false;
    out = ResPlan{};
    ResDims &d = out.d;
    d.n3 = n3;
    d.PS = PS;
    d.colstride = 6LL * n3 * PS;
    d.M = Mt2 * Mt3;
    d.Mt2 = Mt2;
    d.Mt3 = Mt3;
    auto lo = [](int a, int k) { return std::max(a - k, 0); };
    struct L {
        int i2, i3, valid;
    };
    std::vector<std::vector<L>> all(d.M);
    for (int q = 0; q < d.M; ++q) {
        const int a2 = b2[q % Mt2], e2 = b2[q % Mt2 + 1], a3 = b3[q / Mt2], e3 = b3[q / Mt2 + 1];
        ResRank r{};
        r.chunk0 = (int)out.chunks.size();
        for (int type = 0; type < 3; ++type) {
            std::vector<L> v;
            const int x2 = type == 1 ? 2 : 0, x3 = type == 2 ? 2 : 0;
            for (int i3 = lo(a3, x3); i3 < std::min(e3 + x3, n3); ++i3)
                for (int i2 = lo(a2, x2); i2 < std::min(e2 + x2, n2); ++i2) {
                    const bool own = i2 >= a2 && i2 < e2 && i3 >= a3 && i3 < e3;
                    if (type == 0 ? own : !own) v.push_back(L{i2, i3, 1});
                }
            while (v.size() % kResLinesPerChunk) {
                L pad = v.back();
                pad.valid = 0;
                v.push_back(pad);
            }
            out.chunks.insert(out.chunks.end(), v.size() / kResLinesPerChunk, type);
            all[q].insert(all[q].end(), v.begin(), v.end());
            if (type == 0) r.nch0 = (int)out.chunks.size() - r.chunk0;
        }
        r.nch = (int)out.chunks.size() - r.chunk0;
        d.nch0max = std::max(d.nch0max, r.nch0);
        d.nhalomax = std::max(d.nhalomax, r.nch - r.nch0);
        for (const L &l : all[q]) {
            ResLine w;
            w.plo = (l.i3 - lo(a3, 4)) * s.R2 + l.i2 - lo(a2, 4);
            w.f2 = (l.i3 - a3) * s.R2a + l.i2 - lo(a2, 2);
            w.f3 = (l.i3 - lo(a3, 2)) * s.R2b + l.i2 - a2;
            w.info = res_class(l.i2, n2) | res_class(l.i3, n3) << 4 | l.valid << 8;
            out.lines.push_back(w);
            out.gofs.push_back(l.i3 * PS + l.i2 * n1);
        }
        // An iteration's work of a CTA is in its own chunks and, a third as much each, its halo chunks.
        out.cost = std::max(out.cost, d.M * (r.nch0 + (r.nch - r.nch0) / 3.0));
        out.ranks.push_back(r);
    }
    // Who needs which own line: the halo of each CTA, by component. F at the
    // halo rows and the second derivatives reach two lines along both axes;
    // v2 along x2 and v3 along x3 four (F at the second halo row). The places
    // of a line are ordered by direction (along x2, along x3, corners), each
    // direction in columns of its own, so that the lanes of a warp store in
    // step: a tile of eight lines has one place of each kind.
    std::vector<std::vector<std::vector<int>>> dest[3];
    for (auto &v : dest) {
        v.resize(d.M);
        for (int q = 0; q < d.M; ++q) v[q].resize((size_t)out.ranks[q].nch0 * kResLinesPerChunk);
    }
    for (int q = 0; q < d.M; ++q) {
        const int a2 = b2[q % Mt2], e2 = b2[q % Mt2 + 1], a3 = b3[q / Mt2], e3 = b3[q / Mt2 + 1];
        for (int o = 0; o < d.M; ++o) {
            if (o == q) continue;
            const int o2 = o % Mt2, o3 = o / Mt2;
            if (b2[o2] >= e2 + 4 || b2[o2 + 1] + 4 <= a2 || b3[o3] >= e3 + 4 || b3[o3 + 1] + 4 <= a3) continue;
            for (int l = 0; l < out.ranks[o].nch0 * kResLinesPerChunk; ++l) {
                const L &w = all[o][l];
                if (!w.valid) continue;
                const int d2 = w.i2 < a2 ? a2 - w.i2 : w.i2 >= e2 ? w.i2 - e2 + 1 : 0;
                const int d3 = w.i3 < a3 ? a3 - w.i3 : w.i3 >= e3 ? w.i3 - e3 + 1 : 0;
                if (d2 > 4 || d3 > 4) continue;
                int mask = 0;
                if ((d3 == 0 && d2 <= 2) || (d2 == 0 && d3 <= 2)) mask |= 1;
                if (d3 == 0 || (d2 <= 2 && d3 <= 2)) mask |= 2;
                if (d2 == 0 || (d2 <= 2 && d3 <= 2)) mask |= 4;
                const int off = (w.i3 - lo(a3, 4)) * s.R2 + w.i2 - lo(a2, 4);
                if (!mask) continue;
                dest[d3 == 0 ? 0 : d2 == 0 ? 1 : 2][o][l].push_back(q << 28 | mask << 24 | off);
                const int from = o * 3 * s.CS + out.lines[(size_t)out.ranks[o].chunk0 * kResLinesPerChunk + l].plo;
                for (int c = 0; c < 3; ++c)
                    if (mask >> c & 1) out.pull.push_back(ResPull{from + c * s.CS, off + c * s.CS});
            }
        }
        out.ranks[q].npull = (int)out.pull.size() - out.ranks[q].pull0;
        if (q + 1 < d.M) out.ranks[q + 1].pull0 = (int)out.pull.size();
    }
    for (int q = 1; q < d.M; ++q)
        out.ranks[q].push0 = out.ranks[q - 1].push0 + out.ranks[q - 1].nch0 * kResLinesPerChunk;
    int most[3] = {0, 0, 0};
    for (int k = 0; k < 3; ++k)
        for (auto &v : dest[k])
            for (auto &l : v) most[k] = std::max(most[k], (int)l.size());
    d.npush = most[0] + most[1] + most[2];
    for (int q = 0; q < d.M; ++q)
        for (int l = 0; l < out.ranks[q].nch0 * kResLinesPerChunk; ++l)
            for (int k = 0; k < 3; ++k)
                for (int u = 0; u < most[k]; ++u)
                    out.push.push_back(u < (int)dest[k][q][l].size() ? dest[k][q][l][u] : -1);
    if (pull) {
        out.push.clear();
        d.npush = 0;
    }
    d.smem = s.oPush + d.nch0max * kResLinesPerChunk * d.npush * (int)sizeof(int);
    return (size_t)d.smem <= kResSmemMax;
}

// x1 rows: six-point windows from res_start on, in the kernel's parameters.
EQD_HD constexpr int res_start(int i, int n) { return i < 4 ? 0 : (i >= n - 4 ? n - 6 : i - 2); }

// Whether row i of D1 / D2 has a nonzero at entry k of its window (the
// published closures; upper rows mirror the lower ones).
EQD_HD constexpr bool res_nz(bool second, int i, int n, int k) {
    constexpr int d1[5] = {0b001111, 0b000101, 0b011011, 0b110101, 0b011011};
    constexpr int d2[5] = {0b001111, 0b000111, 0b011111, 0b111101, 0b011111};
    const bool up = i >= n - 4;
    const int row = up ? n - 1 - i : (i < 4 ? i : 4);
    return ((second ? d2[row] : d1[row]) >> (up ? 5 - k : k)) & 1;
}

template <typename T, int N1>
struct ResX1 {
    T c1[N1][6], c2[N1][6];  // D1, mu D2
    T hx[N1];                // -hvol times the quadrature weight
};

template <typename T, int N1>
inline ResX1<T, N1> res_x1(double h, double mu, double hvol) {
    ResX1<T, N1> X;
    const Dense1D M(N1, h);
    for (int i = 0; i < N1; ++i) {
        const int s = res_start(i, N1), e = std::min(i, N1 - 1 - i);
        for (int k = 0; k < 6; ++k) {
            X.c1[i][k] = (T)M.d1(i, s + k);
            X.c2[i][k] = (T)(mu * M.d2(i, s + k));
        }
        X.hx[i] = (T)(-hvol * (e < 4 ? kHw[e].v() : 1.0));
    }
    return X;
}

// x2 and x3 rows, one per row class: every row has at most five nonzeros, at
// the own point, its two neighbours and two more (two lines away, or three
// away at the fourth row from an end). A row is read at the offsets off[4]:
//   D1:    c[0..3] at off[0], off[1], off[2], off[3] (its centre is zero, or
//          meets p = 0 on the far-field ring);
//   mu D2: c[4..8] at off[0], -1, 0, 1, off[3] (rows off the ring only);
//   c[9]:  the quadrature weight.
// An unused place has a zero coefficient and the offset of a point that exists.
template <typename T>
inline bool fill_res_tables(int n2, int n3, double h2, double h3, double mu, std::vector<T> &tab, std::vector<int> &off) {
    static const int places[9][4] = {{3, 2, 1, 1},    {-1, -1, 1, 2}, {-2, -1, 1, 2}, {-3, -1, 1, 2}, {-2, -1, 1, 2},
                                     {-1, -1, -2, -3}, {-2, -1, 1, 1}, {-2, -1, 1, 2}, {-2, -1, 1, 3}};
    tab.assign((size_t)18 * kResRow, T(0));
    off.assign(18 * 4, 0);
    for (int a = 0; a < 2; ++a) {
        const int n = a ? n3 : n2;
        const Dense1D M(n, a ? h3 : h2);
        for (int k = 0; k < 9; ++k) {
            const int i = k < 4 ? k : (k == 4 ? 4 : n - 1 - (k - 5)), e = std::min(i, n - 1 - i);
            T *t = &tab[(size_t)(9 * a + k) * kResRow];
            int *o = &off[(size_t)(9 * a + k) * 4];
            std::vector<bool> s1(n, false), s2(n, false);
            for (int c = 0; c < 4; ++c) {
                o[c] = places[k][c];
                const int m = i + o[c];
                if (!s1[m]) t[c] = (T)M.d1(i, m);
                s1[m] = true;
            }
            const int at[5] = {o[0], -1, 0, 1, o[3]};
            for (int c = 0; c < 5 && e > 0; ++c) {
                const int m = i + at[c];
                // a neighbour before the place that repeats it
                const bool again = s2[m] || ((c == 0 || c == 4) && (at[c] == -1 || at[c] == 1));
                if (!again) t[4 + c] = (T)(mu * M.d2(i, m));
                if (!again) s2[m] = true;
            }
            t[9] = (T)(e < 4 ? kHw[e].v() : 1.0);
            for (int m = 0; m < n; ++m) {  // every nonzero has a place
                if (m != i && M.d1(i, m) != 0.0 && !s1[m]) return false;
                if (e > 0 && M.d2(i, m) != 0.0 && !s2[m]) return false;
                if (e > 0 && m == i && M.d1(i, m) != 0.0) return false;
            }
        }
    }
    return true;
}

}  // namespace eqd
