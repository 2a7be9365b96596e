// tma_maps.h -- tensor maps of the TMA-staged D3Q15 steps (host code).
#pragma once

#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

namespace mplb {

// Tensor maps of one kernel over one input population buffer and the
// temperature field (a map holds its box shape, so each kernel has its own).
struct TmaMaps {
    int key = -1;
    const void* f = nullptr;
    const void* T = nullptr;
    alignas(64) CUtensorMap mf;
    alignas(64) CUtensorMap mT;
};

// cuTensorMapEncodeTiled from the driver, found through the runtime (the
// library does not link the driver API).
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// A handle's maps: two kernels x two population buffers.
struct TmaMapCache {
    TmaMaps maps[4];
    int next = 0;
    bool refused = false;  // the driver has no encoder, or refused a map

    // Tensor maps of a step's input buffers: the populations (FP64 or FP32) as a
    // 4D tensor (x, y, z, k) with boxes of bx x by, T as a 3D one (x, y, z) with
    // boxes of tbx x by; no swizzle, zero fill (what lies outside the lattice is
    // written over).  Kept per (key, buffers).  NULL: there are none, and the
    // lattice steps on a kernel without tensor copies.
    const TmaMaps* get(PFN_cuTensorMapEncodeTiled_v12000 enc, int key, int nx, int ny, int nz, const void* fin, bool fp32,
                       const double* Told, uint32_t n, int bx, int by, int tbx) {
        if (refused) return nullptr;
        for (const TmaMaps& m : maps)
            if (m.key == key && m.f == fin && m.T == Told) return &m;
        TmaMaps& m = maps[next];
        const cuuint64_t dims[4] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz, 15};
        auto encode = [&](CUtensorMap* map, bool f32, int rank, const void* p, int width) {
            const cuuint64_t es = f32 ? 4 : 8;
            const cuuint64_t strides[3] = {(cuuint64_t)nx * es, (cuuint64_t)nx * ny * es, (cuuint64_t)n * es};
            const cuuint32_t box[4] = {(cuuint32_t)width, (cuuint32_t)by, 1, 1};
            const cuuint32_t step[4] = {1, 1, 1, 1};
            return enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, rank,
                       const_cast<void*>(p), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
                   CUDA_SUCCESS;
        };
        m.key = -1;
        if (!enc || !encode(&m.mf, fp32, 4, fin, bx) || !encode(&m.mT, false, 3, Told, tbx)) {
            refused = true;
            return nullptr;
        }
        m.key = key;
        m.f = fin;
        m.T = Told;
        next = (next + 1) % 4;
        return &m;
    }
};

}  // namespace mplb
