/*
 * kern_f32_3eq.cu -- kernel configurations of FP32 fields, 3 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(float, CUOPO_F32, 3, 512, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 1024, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 2048, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 1, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 8192, 1, 1, 1),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 4, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 8, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 16, 0, 1),
    CUOPO_K(float, CUOPO_F32, 3, 8192, 16, 1, 1),
};

const KernelList kern_f32_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
