// mplb_march.cu -- instantiations of the marching D2Q9 step (fused_march.cuh),
// compiled without multiply-add contraction like the rest of the FP64 path.
#include <cuda_runtime.h>

#include "fused_march.cuh"

using namespace mplb;

using MarchKernel = void (*)(Params, FusedArgs);

static MarchKernel march_kernel(bool f_on, bool bc) {
    if (f_on) return bc ? k_march_my_d2q9<true, true> : k_march_my_d2q9<true, false>;
    return bc ? k_march_my_d2q9<false, true> : k_march_my_d2q9<false, false>;
}

// Blocks (warps) of the kernel that are resident at once on the current device.
int mplb_march_resident(bool f_on, bool bc) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, march_kernel(f_on, bc), 32, 0);
    return std::max(per, 1) * std::max(sms, 1);
}

cudaError_t mplb_march_launch(bool f_on, bool bc, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    launch_step(march_kernel(f_on, bc), nb, 32, 0, s, P, A);
    return cudaGetLastError();
}
