"""The cells the Verlet-list build walks (`cell_of`, `column_cells`,
quantom_b200/csrc/cellrange.cuh), checked on the host:

* whatever the positions are (inside the box, just outside, far outside,
  infinite, not a number), every run of cells lies inside its column of the
  grid and no length is negative, so the build reads no cell start outside
  [0, m^3];
* for positions inside the box, the runs hold every cell with a point within
  the list radius of a member of the group, once, under the shift that brings it there.

The check is a host program compiled from the header with nvcc (no GPU).
"""
import shutil
import subprocess

import pytest

from conftest import ROOT

CHECK = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "cellrange.cuh"
using namespace lima;

static GroupBox box_of(const std::vector<float>& x, const std::vector<float>& y, const std::vector<float>& z) {
    GroupBox b = {3.4e38f, -3.4e38f, 3.4e38f, -3.4e38f, 3.4e38f, -3.4e38f};   // as the build starts it
    for (size_t p = 0; p < x.size(); p++) {
        if (!(x[p] == x[p])) continue;   // not in the group
        b.xl = fminf(b.xl, x[p]); b.xh = fmaxf(b.xh, x[p]);
        b.yl = fminf(b.yl, y[p]); b.yh = fmaxf(b.yh, y[p]);
        b.zl = fminf(b.zl, z[p]); b.zh = fmaxf(b.zh, z[p]);
    }
    return b;
}

int main() {
    const float nan = nanf(""), inf = INFINITY;
    std::mt19937 rng(5);
    auto uni = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(rng); };
    for (int m : {5, 6, 7, 15}) {
        const float rl = 1.3f, L = 0.5f * rl * (m + 0.4f), cs = L / m, ics = m / L, rl2 = rl * rl;
        std::vector<float> v = {nan, inf, -inf, 3e38f, -3e38f, 1e9f, -1e9f, -990.f, 990.f, -1.f, L + 1.f, 0.f};
        for (int i = -30; i <= 30; i++) v.push_back(0.11f * i * cs);        // near the lower face
        for (int i = -30; i <= 30; i++) v.push_back(L + 0.11f * i * cs);    // near the upper one
        long streams = 0, empty = 0;
        auto check = [&](const std::vector<float>& x, const std::vector<float>& y, const std::vector<float>& z) {
            int hz0 = m, hz1 = -1;
            const int hx = cell_of(x[0], ics, m), hy = cell_of(y[0], ics, m);
            for (size_t p = 0; p < x.size(); p++) {
                const int c = cell_of(z[p], ics, m);
                hz0 = std::min(hz0, c);
                hz1 = std::max(hz1, c);
            }
            if (hx < 0 || hx >= m || hy < 0 || hy >= m || hz0 < 0 || hz1 >= m) { puts("cell"); return false; }
            if (hz1 - hz0 > m - 5) return true;   // not one group
            const GroupBox b = box_of(x, y, z);
            long total = 0;
            for (int k = 0; k < 25; k++) {
                const ColumnCells o = column_cells(k, m, L, cs, ics, rl2, hx, hy, hz0, hz1, b);
                if (o.n0 < 0 || o.n1 < 0 || o.n0 + o.n1 > m) {
                    printf("length %d %d: m %d z %g\n", o.n0, o.n1, m, z[0]);
                    return false;
                }
                for (int r = 0; r < 2; r++) {
                    const int c = r ? o.c1 : o.c0, n = r ? o.n1 : o.n0;
                    if (n && (c < 0 || c + n > m * m * m || c / m != (c + n - 1) / m)) {
                        printf("run %d + %d: m %d z %g\n", c, n, m, z[0]);
                        return false;
                    }
                }
                total += o.n0 + o.n1;
            }
            streams++;
            empty += total == 0;
            return true;
        };
        for (float x : v)
            for (float z : v) {
                if (!check({x}, {0.5f * L}, {z}) || !check({0.5f * L}, {x}, {z}) || !check({x}, {x}, {z})) return 1;
                for (float z2 : {0.5f * L, -7.f * L, 2.f * cs, L - 0.1f * cs})
                    if (!check({0.5f * L, 0.5f * L}, {0.2f * L, 0.2f * L}, {z, z2})) return 1;
            }
        if (!empty || empty == streams) { puts("the positions hold no empty stream"); return 1; }
        // inside the box: all cells in reach, each under its own image
        for (int t = 0; t < 300; t++) {
            std::vector<float> x, y, z;
            const int hx = rng() % m, hy = rng() % m, h0 = rng() % m, h1 = std::min(m - 1, h0 + (int)(rng() % (m - 4)));
            for (int p = 0; p < 3; p++) {
                x.push_back(uni(hx * cs * 1.0001f, (hx + 0.999f) * cs));
                y.push_back(uni(hy * cs * 1.0001f, (hy + 0.999f) * cs));
                z.push_back(uni(h0 * cs * 1.0001f, (h1 + 0.999f) * cs));
            }
            int hz0 = m, hz1 = -1;
            for (float c : z) hz0 = std::min(hz0, cell_of(c, ics, m)), hz1 = std::max(hz1, cell_of(c, ics, m));
            const GroupBox b = box_of(x, y, z);
            std::vector<int> seen(m * m * m, 0);
            std::vector<float> sx(m * m * m), sy(m * m * m), sz(m * m * m);
            for (int k = 0; k < 25; k++) {
                const ColumnCells o = column_cells(k, m, L, cs, ics, rl2, hx, hy, hz0, hz1, b);
                for (int r = 0; r < 2; r++)
                    for (int c = r ? o.c1 : o.c0, e = c + (r ? o.n1 : o.n0); c < e; c++) {
                        seen[c]++;
                        sx[c] = o.sx;
                        sy[c] = o.sy;
                        sz[c] = r ? o.sz1 : o.sz0;
                    }
            }
            for (int c : seen)
                if (c > 1) { puts("a cell twice"); return 1; }
            for (int q = 0; q < 4000; q++) {   // a point within the list radius of a member
                const int p = rng() % 3;
                const float r = rl * 0.999f * cbrtf(uni(0.f, 1.f)), ct = uni(-1.f, 1.f), ph = uni(0.f, 6.2831853f);
                const float st = sqrtf(1.f - ct * ct);
                const float ux = x[p] + r * st * cosf(ph), uy = y[p] + r * st * sinf(ph), uz = z[p] + r * ct;
                float w[3] = {ux, uy, uz};
                for (float& a : w) a += a < 0.f ? L : (a >= L ? -L : 0.f);
                if (w[0] >= L || w[1] >= L || w[2] >= L) continue;   // rounded onto the face
                const int c = (cell_of(w[0], ics, m) * m + cell_of(w[1], ics, m)) * m + cell_of(w[2], ics, m);
                if (!seen[c]) { printf("missed cell: m %d z %g + %g\n", m, z[p], r * ct); return 1; }
                if (fabsf(w[0] + sx[c] - ux) > 1e-3f || fabsf(w[1] + sy[c] - uy) > 1e-3f || fabsf(w[2] + sz[c] - uz) > 1e-3f) {
                    puts("wrong image");
                    return 1;
                }
            }
        }
    }
    puts("ok");
    return 0;
}
"""


def test_walked_cells_lie_in_the_grid_and_cover_the_reach(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "check.cu"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    cmd = [nvcc, "-std=c++17", "-O2", f"-I{ROOT / 'quantom_b200' / 'csrc'}", str(src), "-o", str(exe),
           "-Wno-deprecated-gpu-targets"]
    subprocess.run(cmd, check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
