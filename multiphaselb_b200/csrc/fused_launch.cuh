// fused_launch.cuh -- launches of the general fused kernels by tile candidate.
// Included by the translation unit of the steps without surface tension
// (fused_host.cuh) and by that of the steps with it (mplb_st.cu), each of which
// instantiates its own kernels; both are compiled without multiply-add
// contraction.
#pragma once

#include "fused.cuh"

namespace mplb {

template <int TX, int TY, bool PIPE, bool HAS_BC, bool EMIT, bool ST = false>
cudaError_t set_smem3() {
    if constexpr (PIPE)
        return cudaFuncSetAttribute(k_fused_d3q15_pipe<TX, TY, HAS_BC, EMIT, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)f3_smem<TX, TY, PIPE>());
    else
        return cudaFuncSetAttribute(k_fused_d3q15<TX, TY, HAS_BC, EMIT, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)f3_smem<TX, TY, PIPE>());
}

// The 3D kernels use more than the 48 KB of static shared memory.
template <bool ST>
cudaError_t general_attributes() {
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
#define MPLB_SET3(TX, TY, PIPE) chk(set_smem3<TX, TY, PIPE, true, false, ST>()); chk(set_smem3<TX, TY, PIPE, false, false, ST>());
    MPLB_SET3(32, 8, false)
    MPLB_SET3(32, 8, true)
    MPLB_SET3(32, 4, false)
    MPLB_SET3(64, 4, false)
    MPLB_SET3(32, 16, false)
#undef MPLB_SET3
    return e;
}

template <int TX, int TY, int MINB, bool F_ON, bool G_ON, bool EMIT, bool INNER, bool MY = false, int RINGW = 0,
          bool ST = false>
void launch2(bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    constexpr int nt = TX * TY + 32 * RINGW;
    if (bc) launch_step(k_fused_d2q9<TX, TY, MINB, F_ON, G_ON, true, EMIT, INNER, MY, RINGW, ST>, nb, nt, 0, s, P, A);
    else launch_step(k_fused_d2q9<TX, TY, MINB, F_ON, G_ON, false, EMIT, INNER, MY, RINGW, ST>, nb, nt, 0, s, P, A);
}

// A lattice with a surface-tension term (ST) updates its flow.
template <int TX, int TY, bool EMIT, int MINB = 0, bool INNER = false, int RINGW = 0, bool ST = false>
void launch2_fg(bool fon, bool gon, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    const bool my = gon && P.g_model == MPLB_MYMRT;
    if (fon && my) launch2<TX, TY, MINB, true, true, EMIT, INNER, true, RINGW, ST>(bc, nb, P, A, s);
    else if (fon && gon) launch2<TX, TY, MINB, true, true, EMIT, INNER, false, RINGW, ST>(bc, nb, P, A, s);
    else if (fon) launch2<TX, TY, MINB, true, false, EMIT, INNER, false, RINGW, ST>(bc, nb, P, A, s);
    if constexpr (!ST) {
        if (!fon && my) launch2<TX, TY, MINB, false, true, EMIT, INNER, true, RINGW>(bc, nb, P, A, s);
        else if (!fon && gon) launch2<TX, TY, MINB, false, true, EMIT, INNER, false, RINGW>(bc, nb, P, A, s);
    }
}

template <int TX, int TY, bool PIPE, bool EMIT, bool ST = false>
void launch3(bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    constexpr size_t sm = f3_smem<TX, TY, PIPE>();
    if constexpr (PIPE) {
        if (bc) launch_step(k_fused_d3q15_pipe<TX, TY, true, EMIT, ST>, nb, TX * TY, sm, s, P, A);
        else launch_step(k_fused_d3q15_pipe<TX, TY, false, EMIT, ST>, nb, TX * TY, sm, s, P, A);
    } else {
        if (bc) launch_step(k_fused_d3q15<TX, TY, true, EMIT, ST>, nb, TX * TY, sm, s, P, A);
        else launch_step(k_fused_d3q15<TX, TY, false, EMIT, ST>, nb, TX * TY, sm, s, P, A);
    }
}

// One step of 2D candidate `cfg` (a tile kernel).
template <bool ST>
void launch_general2(int cfg, bool f_on, bool g_on, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    switch (cfg) {
    case 0: launch2_fg<32, 8, false, 0, false, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 1: launch2_fg<32, 4, false, 0, false, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 2: launch2_fg<64, 4, false, 0, false, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 3: launch2_fg<16, 8, false, 0, true, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 4: launch2_fg<64, 4, false, 0, true, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 5: launch2_fg<16, 8, false, 6, true, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 6: launch2_fg<32, 8, false, 3, true, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 7: launch2_fg<32, 4, false, 8, true, 0, ST>(f_on, g_on, bc, nb, P, A, s); break;
    case 8: launch2_fg<32, 8, false, 2, false, 3, ST>(f_on, g_on, bc, nb, P, A, s); break;
    default: launch2_fg<16, 8, false, 4, false, 2, ST>(f_on, g_on, bc, nb, P, A, s); break;
    }
}

// One step of 3D candidate `cfg` (a tile kernel without TMA).
template <bool ST>
void launch_general3(int cfg, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    switch (cfg) {
    case 0: launch3<32, 8, false, false, ST>(bc, nb, P, A, s); break;
    case 1: launch3<32, 8, true, false, ST>(bc, nb, P, A, s); break;
    case 2: launch3<32, 4, false, false, ST>(bc, nb, P, A, s); break;
    case 3: launch3<64, 4, false, false, ST>(bc, nb, P, A, s); break;
    default: launch3<32, 16, false, false, ST>(bc, nb, P, A, s); break;
    }
}

}  // namespace mplb
