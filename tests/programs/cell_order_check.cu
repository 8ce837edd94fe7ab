// Checks parm::cell_row and parm::cell_coords (parm_gb300/csrc/parm_internal.cuh)
// on the host: over grids and tile widths, with remainders and with one tile,
// every cell of a grid has its own index below the cell count and cell_coords
// gives the cell of that index back; prints "ok <count>" or the first mismatch.
// Test infrastructure.
#include <cstdio>
#include <vector>

#include "parm_internal.cuh"

int main() {
    long count = 0;
    for (int nx : {1, 2, 5})
        for (int ny : {1, 3, 4, 5, 8, 9, 31})
            for (int nz : {1, 3, 7})
                for (uint32_t tile : {1u, 2u, 4u, 5u, 30u, 31u, 64u}) {
                    parm::SysConst S{};
                    S.nc[0] = nx, S.nc[1] = ny, S.nc[2] = nz, S.ytile = tile;
                    std::vector<int> seen(nx * ny * nz, 0);
                    for (int z = 0; z < nz; z++)
                        for (int y = 0; y < ny; y++)
                            for (int x = 0; x < nx; x++, count++) {
                                const uint32_t b = parm::cell_row(S, y, z) * (uint32_t)nx + (uint32_t)x;
                                uint32_t c[3] = {~0u, ~0u, ~0u};
                                if (b < seen.size()) parm::cell_coords(S, b, c);
                                if (b >= seen.size() || seen[b]++ || c[0] != (uint32_t)x || c[1] != (uint32_t)y ||
                                    c[2] != (uint32_t)z) {
                                    std::printf("grid %d %d %d tile %u cell %d %d %d: index %u\n", nx, ny, nz, tile, x,
                                                y, z, b);
                                    return 1;
                                }
                            }
                }
    std::printf("ok %ld\n", count);
    return 0;
}
