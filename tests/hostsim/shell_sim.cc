// The work items of the periodic image copies (shell_cell, dev_common.cuh)
// against a walk over the whole box: the same cells with the same images,
// each once, for every mix of periodic and walled axes and both tables.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>

#include <cuda_runtime.h>
#include <strings.h>

inline int __ffs(int v) { return ffs(v); }

#include "dev_common.cuh"

using namespace rmt3d;

int main() {
    const int sizes[][3] = {{4, 5, 6}, {8, 4, 4}, {5, 9, 7}};
    for (auto &n : sizes)
        for (int p = 0; p < 8; p++)
            for (int corner = 0; corner < 2; corner++) {
                grid_dev g;
                memset(&g, 0, sizeof(g));
                g.sm = n[0], g.sn = n[1], g.so = n[2];
                g.sm4 = g.sm + 4, g.sn4 = g.sn + 4, g.so4 = g.so + 4, g.smn4 = g.sm4 * g.sn4, g.ncell = g.smn4 * g.so4;
                for (int d = 0; d < 3; d++) g.prd[d] = (p >> d) & 1;
                std::map<int, int> want, got;
                for (int k = 0; k < g.so4; k++)
                    for (int j = 0; j < g.sn4; j++)
                        for (int i = 0; i < g.sm4; i++) {
                            const int c[3] = {i, j, k};
                            int m[3];
                            bool ghost = false, ok = true;
                            for (int d = 0; d < 3; d++) {
                                const int len = n[d] + (corner && !g.prd[d] ? 1 : 0);
                                m[d] = c[d];
                                if (c[d] >= 2 && c[d] < 2 + len) continue;
                                if (!g.prd[d]) ok = false;
                                ghost = true;
                                m[d] += c[d] < 2 ? n[d] : -n[d];
                            }
                            if (ok && ghost) want[gidx(g, i, j, k)] = gidx(g, m[0], m[1], m[2]);
                        }
                const int cells = shell_cells(g, corner);
                for (int t = 0; t < cells; t++) {
                    int dst, src;
                    if (!shell_cell(g, corner, t, dst, src)) continue;
                    if (dst < 0 || dst >= g.ncell || src < 0 || src >= g.ncell || got.count(dst)) return 2;
                    got[dst] = src;
                }
                if (got != want) {
                    printf("axes %d corner %d: %zu cells, want %zu\n", p, corner, got.size(), want.size());
                    return 1;
                }
            }
    return 0;
}
