// Host-only check of the marching kernel's index arithmetic (no GPU needed):
// every node is finished by exactly one lane, and every column, row and pull
// source a lane forms lies in the box and is the one pull_src gives.
// Prints "OK <cases>" or the first violation.
#include <cstdio>
#include <vector>
#include "../multiphaselb_b200/csrc/fused_march.cuh"

using namespace mplb;

int main() {
    int cases = 0, fails = 0;
#define REQUIRE(c, ...) do { if (!(c) && fails++ < 10) { printf("FAIL %s:%d ", __FILE__, __LINE__); printf(__VA_ARGS__); printf("\n"); } } while (0)
    const int dims[][2] = {{2, 2}, {2, 9}, {27, 5}, {28, 28}, {29, 31}, {56, 4}, {57, 97}, {128, 512}, {1021, 63}};
    for (auto& d : dims)
        for (int per = 0; per < 4; per++)
            for (int resident : {1, 148, 1776}) {
                FusedArgs A{};
                A.nx = d[0]; A.ny = d[1]; A.nz = 1; A.px = per & 1; A.py = per >> 1; A.pz = 1;
                const Geom g = march_geometry(A, resident);
                std::vector<int> owned((size_t)A.nx * A.ny, 0);
                for (int b = 0; b < g.nblocks; b++) {
                    const int strip = b % g.tiles_x, chunk = b / g.tiles_x;
                    const int y0 = chunk * g.zchunk, y1 = std::min(y0 + g.zchunk, A.ny);
                    REQUIRE(y0 < A.ny, "empty chunk %d", chunk);
                    for (int lane = 0; lane < 32; lane++) {
                        const int xo = strip * MARCH_W - MARCH_H + lane;
                        const int xw = xo < A.nx + MARCH_H ? march_wrap(xo, A.nx, A.px) : -1;
                        if (xw < 0) continue;
                        REQUIRE(xw < A.nx, "column %d of %d", xw, A.nx);
                        const int xl = march_wrap(xw - 1, A.nx, A.px), xr = march_wrap(xw + 1, A.nx, A.px);
                        for (int j = y0 - MARCH_H; j < y1 + MARCH_H; j++) {
                            const int y = march_wrap(j, A.ny, A.py);
                            if (y < 0) continue;
                            REQUIRE(y < A.ny, "row %d of %d", y, A.ny);
                            const int yd = march_wrap(y - 1, A.ny, A.py), yu = march_wrap(y + 1, A.ny, A.py);
                            for (int k = 0; k < 9; k++) {
                                const int cx = cxk<D2Q9T>(k), cy = cyk<D2Q9T>(k);
                                const int sx = cx == 1 ? xl : (cx == -1 ? xr : xw), sy = cy == 1 ? yd : (cy == -1 ? yu : y);
                                const long got = sx < 0 || sy < 0 ? -1 : (long)sx + (long)A.nx * sy;
                                REQUIRE(got == pull_src(A.nx, A.ny, 1, A.px, A.py, 1, xw, y, 0, cx, cy, 0), "source k %d", k);
                            }
                            const int e = j;  // the row is finished two rows later
                            if (e >= y0 && e < y1 && lane >= MARCH_H && lane < 32 - MARCH_H && xo >= 0 && xo < A.nx)
                                owned[(size_t)xo + (size_t)A.nx * e]++;
                        }
                    }
                }
                for (size_t i = 0; i < owned.size(); i++) REQUIRE(owned[i] == 1, "node %zu owned %d times", i, owned[i]);
                cases++;
            }
    if (fails) { printf("FAILED %d checks\n", fails); return 1; }
    printf("OK %d\n", cases);
    return 0;
}
