/*
 * kern_f32_3eq.cu -- kernel configurations of FP32 fields, 3 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(float, CUOPO_F32, 3, 512, 1, 0, 1, 6.7, 10),
    CUOPO_K(float, CUOPO_F32, 3, 1024, 1, 0, 1, 6.9, 10.2),
    CUOPO_K(float, CUOPO_F32, 3, 2048, 1, 0, 1, 7.7, 10.7),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 1, 0, 1, 11.8, 11.8),
    /* 2^13: two in-place CTAs per SM run 148 instances in 24.1 us per slice, the
     * single 8192-point CTA 27.5 (kept for callers that need one CTA) */
    CUOPO_K(float, CUOPO_F32, 3, 4096, 2, 1, 2, 16.8, 24.1),
    CUOPO_K(float, CUOPO_F32, 3, 8192, 1, 1, 1, 0, 0),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 4, 0, 1, 17.2, 17.2),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 8, 0, 1, 20.1, 20.1),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 16, 0, 1, 23.9, 23.9),
    CUOPO_K(float, CUOPO_F32, 3, 8192, 16, 1, 1, 0, 0),
};

const KernelList kern_f32_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
