/*
 * kern_f32_2eq.cu -- kernel configurations of FP32 fields, 2 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(float, CUOPO_F32, 2, 512, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 1024, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 2048, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 1, 0, 2),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 2, 0, 2),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 4, 0, 2),
    CUOPO_K(float, CUOPO_F32, 2, 4096, 8, 0, 2),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 2, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 4, 0, 1),
    CUOPO_K(float, CUOPO_F32, 2, 8192, 8, 0, 1),
};

const KernelList kern_f32_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
