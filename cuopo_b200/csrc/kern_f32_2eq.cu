/*
 * kern_f32_2eq.cu -- kernel configurations of FP32 fields, 2 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(float, CUOPO_F32, 2, 512, 1, 0, 1, 7, 9.4),
    CUOPO_K(float, CUOPO_F32, 2, 1024, 1, 0, 1, 7.3, 9.4),
    CUOPO_K(float, CUOPO_F32, 2, 2048, 1, 0, 1, 7.9, 9.8),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 1, 0, 2, 11.1, 17.9),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 2, 0, 2, 13.9, 20.7),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 1, 0, 1, 0, 0),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 4, 0, 2, 14.6, 24.3),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 8, 0, 2, 16.8, 27),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 2, 0, 1, 0, 0),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 4, 0, 1, 0, 0),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 8, 0, 1, 0, 0),
};

const KernelList kern_f32_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
