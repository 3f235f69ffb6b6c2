/*
 * wide_f32_2eq.cu -- other layouts of the configurations of kern_f32_2eq.cu.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(float, CUOPO_F32, 2, 512, 1, 1, 128, 1, 1, 2.95, 4.3),
    CUOPO_W(float, CUOPO_F32, 2, 512, 1, 2, 128, 2, 4, 2.5, 3.1),
    CUOPO_W(float, CUOPO_F32, 2, 1024, 1, 1, 256, 1, 1, 3.4, 3.5),
    CUOPO_W(float, CUOPO_F32, 2, 1024, 1, 4, 128, 2, 4, 2.6, 3.3),
    CUOPO_W(float, CUOPO_F32, 2, 2048, 1, 1, 256, 1, 1, 5.3, 5.3),
    CUOPO_W(float, CUOPO_F32, 2, 2048, 1, 4, 128, 1, 1, 4, 4.6),
    CUOPO_W(float, CUOPO_F32, 2, 2048, 1, 8, 128, 2, 4, 3.1, 3.2),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 1, 2, 256, 1, 1, 7.1, 7.1),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 1, 4, 256, 1, 1, 4.2, 4.2),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 1, 16, 128, 2, 4, 3.2, 3.3),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 2, 4, 256, 1, 1, 7.4, 7.4),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 2, 8, 256, 1, 1, 5, 5),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 2, 16, 256, 1, 1, 3.5, 3.5),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 4, 8, 256, 1, 1, 8.2, 8.2),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 4, 16, 256, 1, 1, 5.1, 5.1),
    CUOPO_W(float, CUOPO_F32, 2, 4096, 8, 16, 256, 1, 1, 8.4, 8.4),
};

const KernelList wide_f32_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
