// The cell grid of the physics path and the cells that the list build walks,
// as plain functions of positions (host and device, so that the index
// arithmetic can be checked without a GPU).
#pragma once
#include <cmath>

#include <cuda_runtime.h>

namespace lima {

__host__ __device__ inline int min_i(int a, int b) { return a < b ? a : b; }
__host__ __device__ inline int max_i(int a, int b) { return a > b ? a : b; }

// cell of a coordinate (inv: cells per length), clamped to the grid (cell 0 for what is not a number)
__host__ __device__ inline int cell_of(float x, float inv, int m) {
    return (int)fminf(fmaxf(x * inv, 0.f), (float)(m - 1));
}

// bounding box of a group of particles that share a home column
struct GroupBox {
    float xl, xh, yl, yh, zl, zh;
};

// Up to two runs of consecutive cells of one column, with the shifts that
// bring their particles into the group's home frame.
struct ColumnCells {
    int c0, n0;   // first run: its first cell (in the grid) and its cells
    int c1, n1;
    float sx, sy, sz0, sz1;
};

// Column k (0 .. 24) of the 5 x 5 columns around home column (hx, hy): the
// cells that the group's particles (in cells hz0 .. hz1 of the home column,
// hz1 - hz0 <= m - 5, m >= 5) can reach within the list radius, none where the
// xy gap between the group and the column exceeds it.
__host__ __device__ inline ColumnCells column_cells(int k, int m, float L, float cs, float ics, float rlist2, int hx,
                                                    int hy, int hz0, int hz1, const GroupBox& b) {
    ColumnCells o = {0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f};
    const int ox = k / 5 - 2, oy = k % 5 - 2;
    const float cxl = (float)(hx + ox) * cs, cxh = cxl + cs;   // unwrapped, home frame
    const float cyl = (float)(hy + oy) * cs, cyh = cyl + cs;
    const float gx = fmaxf(0.f, fmaxf(cxl - b.xh, b.xl - cxh));
    const float gy = fmaxf(0.f, fmaxf(cyl - b.yh, b.yl - cyh));
    const float g2 = gx * gx + gy * gy;
    if (g2 < rlist2 * 1.0001f) {   // the margin covers cell rounding
        int x = hx + ox, y = hy + oy;
        if (x < 0) { x += m; o.sx = -L; } else if (x >= m) { x -= m; o.sx = L; }
        if (y < 0) { y += m; o.sy = -L; } else if (y >= m) { y -= m; o.sy = L; }
        const int col = (x * m + y) * m;
        // cells within the reach of the group's z-range (unwrapped; at most m
        // of them: the group spans <= m - 4 cells)
        const float reach = sqrtf(fmaxf(rlist2 - g2, 0.f)) + 1e-4f * cs;
        const int lo = hz0 - 2, hi = hz1 + 2;
        const int u0 = (int)fminf(fmaxf(floorf((b.zl - reach) * ics), (float)lo), (float)hi);
        const int u1 = (int)fmaxf(fminf(floorf((b.zh + reach) * ics), (float)hi), (float)(u0 - 1));
        // below the grid, inside it, above it: the parts below and above hold
        // cells of the far end, and the span leaves at most two of the three
        // parts (none where a particle far outside the box has u1 < u0)
        const int in0 = max_i(u0, 0), in1 = min_i(u1, m - 1);
        o.n0 = o.n1 = max_i(in1 - in0 + 1, 0);
        if (u0 < 0) {
            o.c0 = col + u0 + m;
            o.n0 = max_i(min_i(u1, -1) - u0 + 1, 0);
            o.sz0 = -L;
            o.c1 = col;
        } else {
            o.c0 = col + in0;
            o.c1 = col + max_i(u0 - m, 0);
            o.n1 = max_i(u1 - max_i(u0, m) + 1, 0);
            o.sz1 = L;
        }
    }
    return o;
}

}  // namespace lima
