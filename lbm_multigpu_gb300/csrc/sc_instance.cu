/*
 * sc_instance.cu -- the stream-collide kernels (sc_kernels.cuh) of one storage
 * format and population layout, chosen by the build: LBM_SC_TYPE (its element
 * type), LBM_SC_NAME (f32, f16, bf16, f64) and LBM_SC_LAY (0: structure of
 * arrays, 1: blocks of 32 nodes with each opposite pair interleaved).
 */
#include "sc_kernels.cuh"

#define LBM_CAT_(a, b, c) a##b##_##c
#define LBM_CAT(a, b, c) LBM_CAT_(a, b, c)

namespace lbm {

cudaError_t LBM_CAT(launch_sc_, LBM_SC_NAME, LBM_SC_LAY)(const Level& L, const StepParams& p, const void* fA, void* fB,
                                                         const uint8_t* mask, float* stats, float* mom_export,
                                                         cudaStream_t s, const uint32_t* links) {
    return launch_sc_t<LBM_SC_TYPE, LBM_SC_LAY>(L, p, fA, fB, mask, stats, mom_export, s, links);
}

cudaError_t LBM_CAT(launch_sc_mlp_, LBM_SC_NAME, LBM_SC_LAY)(const Level& L, const StepParams& p, const void* fA,
                                                             void* fB, const uint8_t* mask, float* stats,
                                                             const uint32_t* links, const void* blob, int* err,
                                                             cudaStream_t s) {
    /* the closure's arithmetic is FP32 */
    if constexpr (sizeof(LBM_SC_TYPE) <= 4)
        return launch_sc_mlp_t<LBM_SC_TYPE, LBM_SC_LAY>(L, p, fA, fB, mask, stats, links, blob, err, s);
    else
        return cudaErrorInvalidValue;
}

}  // namespace lbm
