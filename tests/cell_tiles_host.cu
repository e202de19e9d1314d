// The tiles of the kernels over cells (cell_grid, isf_common.cuh): for every
// nx ny pair read, how often each cell of a plane is covered (all once: "ok")
// and the lanes a plane takes.  Built and driven by test_cell_tiles_cpu.py.
#include <cstdio>
#include <vector>

#include "isf_common.cuh"

int main() {
    int nx, ny;
    while (std::scanf("%d %d", &nx, &ny) == 2) {
        isf::Grid g = {};
        g.n[0] = nx, g.n[1] = ny, g.n[2] = 1;
        g.ctw = isf::cell_tile_width(nx, ny);
        const dim3 grid = isf::cell_grid(g);
        std::vector<int> seen(nx * ny, 0);
        for (int by = 0; by < (int)grid.y; ++by)
            for (int bx = 0; bx < (int)grid.x; ++bx)
                for (int t = 0; t < 256; ++t) {
                    const int x = isf::cell_x(g, bx, t), y = isf::cell_y(g, by, t);
                    if (x < nx && y < ny) ++seen[x + nx * y];
                }
        bool ok = true;
        for (int n : seen) ok = ok && n == 1;
        std::printf("%s %d\n", ok ? "ok" : "bad", (int)(grid.x * grid.y * 256));
    }
}
