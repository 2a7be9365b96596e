// Host-only check of the FP32 D3Q15 step's choice of its kernel by the box's
// extents (no GPU needed).  Prints "OK", or the first violation.
#include <cstdio>
#include "../multiphaselb_b200/csrc/fused32_tma.cuh"

using namespace mplb;

#define REQUIRE(c, ...) do { if (!(c)) { printf("FAIL line %d ", __LINE__); printf(__VA_ARGS__); printf("\n"); return 1; } } while (0)

int main() {
    // blocks per SM of the general kernel
    const int four[][3] = {{250, 230, 8}, {250, 250, 2}, {250, 250, 4}, {250, 250, 8}, {60, 60, 128}, {250, 290, 8},
                           {192, 192, 10}, {256, 160, 10}, {256, 160, 12}};
    const int five[][3] = {{100, 60, 33}, {130, 130, 16}, {250, 200, 8}, {300, 240, 4}, {130, 130, 33}, {97, 61, 83},
                           {101, 75, 90}, {150, 150, 150}, {256, 256, 12}};
    auto blocks = [](const int* d) {
        FusedArgs A{};
        A.nx = d[0]; A.ny = d[1]; A.nz = d[2];
        return general32_blocks(fused_geometry(MPLB_D3Q15, A, 32, 4), d[2]);
    };
    for (auto& d : four) REQUIRE(blocks(d) == 4, "%d x %d x %d: %d", d[0], d[1], d[2], blocks(d));
    for (auto& d : five) REQUIRE(blocks(d) == 5, "%d x %d x %d: %d", d[0], d[1], d[2], blocks(d));
    // the general kernel (-1) or the TMA-staged one (0: 64 x 8 tiles, 1: 32 x 8): boxes whose
    // kernels differ by more than 5 %, and none but a kernel that takes the box
    auto tile = [](const int* d, bool bc = false) {
        FusedArgs A{};
        A.nx = d[0]; A.ny = d[1]; A.nz = d[2]; A.px = A.py = A.pz = 1;
        return tma32_tile(A, bc);
    };
    const int general[][3] = {{32, 8, 2}, {32, 8, 7}, {64, 8, 4}, {64, 8, 7}, {64, 16, 3}, {32, 32, 6}, {64, 64, 4}, {96, 64, 5},
                              {128, 128, 2}, {128, 128, 6}, {96, 160, 4}, {192, 192, 4}, {256, 160, 6}, {320, 256, 2},
                              {320, 256, 8}, {320, 320, 2}, {320, 320, 5}, {512, 512, 2}};
    const int tma64[][3] = {{192, 192, 8}, {128, 128, 128}, {192, 192, 192}, {256, 256, 16}};
    const int tma32[][3] = {{32, 8, 8}, {64, 8, 16}, {64, 16, 8}, {32, 32, 16}, {64, 64, 16}, {96, 64, 24}, {128, 128, 8},
                            {96, 160, 16}, {96, 96, 96}};
    for (auto& d : general) REQUIRE(tile(d) == -1, "%d x %d x %d: %d", d[0], d[1], d[2], tile(d));
    for (auto& d : tma64) REQUIRE(tile(d) == 0, "%d x %d x %d: %d", d[0], d[1], d[2], tile(d));
    for (auto& d : tma32) REQUIRE(tile(d) == 1, "%d x %d x %d: %d", d[0], d[1], d[2], tile(d));
    for (int nx = 2; nx <= 200; nx += 7)
        for (int ny = 2; ny <= 80; ny += 3)
            for (int nz : {2, 5, 8, 40}) {
                const int d[3] = {nx, ny, nz}, t = tile(d);
                REQUIRE(t == -1 || (ny % 8 == 0 && nx % (t == 0 ? 64 : 32) == 0), "%d x %d x %d: %d", nx, ny, nz, t);
                REQUIRE(tile(d, true) == -1, "boundary programs");
            }
    printf("OK\n");
    return 0;
}
