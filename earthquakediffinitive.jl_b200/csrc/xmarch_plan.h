// Host-side plan of the x1 march (xmarch.cuh): the length of a stored x2 line,
// the tiles of an axis, and the columns that the kernel can address.
#pragma once
#include <algorithm>
#include <vector>

namespace eqd {

constexpr int kXLead = 3;  // x2 line i2 is stored at kXLead + i2

inline int x_row_length(int n2) { return (n2 + kXLead + 3) / 4 * 4; }

// Elements of a column.
inline long long x_column(int n1, int n2, int n3) { return 6LL * n1 * n3 * x_row_length(n2); }

// Whether every byte of a column has a 32-bit offset from its start: the march
// keeps a line's place, and the steps from x to x and from component to
// component, as 32-bit byte offsets. A column of more than 2^30 elements (21 x
// 3201 x 3201 nodes a side) streams x1-fastest.
inline bool x_offsets_fit(int n1, int n2, int n3) { return 4 * x_column(n1, n2, n3) <= 1LL << 32; }

// Tile bounds along an axis of n nodes, at most `width` lines a tile,
// from `first` to n - 1 in multiples of `step`, as few tiles as possible. A
// tile sees two lines of F and four of p beyond its own: no inner bound may
// have a closure row that reaches further (rows 0 .. 3 read up to row 5, row 3
// three lines back).
inline bool x_tiles(int n, int first, int width, int step, std::vector<int> &b) {
    const int end = n - 1;
    std::vector<int> best(end + 1, 1 << 20), from(end + 1, -1);
    best[first] = 0;
    for (int e = first + 1; e <= end; ++e) {
        if (e < end && ((e - first) % step || e < 4 || e > n - 4 || e == 5 || e == n - 5)) continue;
        for (int a = std::max(first, e - width); a < e; ++a)
            if (best[a] + 1 < best[e]) {
                best[e] = best[a] + 1;
                from[e] = a;
            }
    }
    if (best[end] >= 1 << 20) return false;
    b.clear();
    for (int e = end; e != first; e = from[e]) b.push_back(e);
    b.push_back(first);
    std::reverse(b.begin(), b.end());
    return true;
}

}  // namespace eqd
