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
                           {101, 75, 90}, {150, 150, 150}};
    auto blocks = [](const int* d) {
        FusedArgs A{};
        A.nx = d[0]; A.ny = d[1]; A.nz = d[2];
        return general32_blocks(fused_geometry(MPLB_D3Q15, A, 32, 4), d[2]);
    };
    for (auto& d : four) REQUIRE(blocks(d) == 4, "%d x %d x %d: %d", d[0], d[1], d[2], blocks(d));
    for (auto& d : five) REQUIRE(blocks(d) == 5, "%d x %d x %d: %d", d[0], d[1], d[2], blocks(d));
    printf("OK\n");
    return 0;
}
