// mplb_st.cu -- the general fused steps of lattices with a surface-tension term,
// every tile candidate (fused_launch.cuh), compiled without multiply-add
// contraction.
#include <cuda_runtime.h>

#include "fused_launch.cuh"

using namespace mplb;

cudaError_t mplb_st_attributes() { return general_attributes<true>(); }

void mplb_st_launch2(int cfg, bool g_on, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    launch_general2<true>(cfg, true, g_on, bc, nb, P, A, s);
}

void mplb_st_launch3(int cfg, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    launch_general3<true>(cfg, bc, nb, P, A, s);
}
