// Host-only check of the FP32 D3Q15 step's choice between the TMA-staged kernel
// and the general one when tensor maps cannot be had (no GPU needed; stand-ins
// for the driver's encoder).  Prints "OK", or the first violation.
#include <cstdio>
#include "../multiphaselb_b200/csrc/fused32_tma.cuh"

using namespace mplb;

static int calls = 0, fail_from = 0;  // the encoder's calls; the first one that fails (0: none)
static CUresult CUDAAPI encoder(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return ++calls >= fail_from && fail_from ? CUDA_ERROR_INVALID_VALUE : CUDA_SUCCESS;
}

#define REQUIRE(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    FusedArgs A{};
    A.nx = 192; A.ny = 192; A.nz = 192; A.px = A.py = A.pz = 1;
    const uint32_t n = 192u * 192u * 192u;
    static float f[2][4];
    static double T[4];
    {
        TmaMapCache c;  // maps are kept per buffer
        for (int step = 0; step < 4; step++) {
            const Tma32 t = tma32_choose(c, encoder, A, false, n, f[step & 1], T);
            REQUIRE(t.tile >= 0 && t.maps && t.maps->f == f[step & 1]);
        }
        REQUIRE(calls == 4);
        REQUIRE(tma32_choose(c, encoder, A, true, n, f[0], T).tile == -1);  // boundary programs
        REQUIRE(!c.refused);
    }
    {
        TmaMapCache c;  // no encoder in the driver
        REQUIRE(tma32_choose(c, nullptr, A, false, n, f[0], T).tile == -1);
        REQUIRE(tma32_choose(c, nullptr, A, false, n, f[1], T).tile == -1);
    }
    for (fail_from = 1; fail_from <= 4; fail_from++) {  // the first or the second map of either buffer refused
        TmaMapCache c;
        calls = 0;
        const Tma32 a = tma32_choose(c, encoder, A, false, n, f[0], T), b = tma32_choose(c, encoder, A, false, n, f[1], T);
        REQUIRE((a.tile >= 0) == (fail_from > 2) && b.tile == -1 && !b.maps);
        const int asked = calls;
        REQUIRE(tma32_choose(c, encoder, A, false, n, f[0], T).tile == -1 && calls == asked);  // not asked again
    }
    printf("OK\n");
    return 0;
}
