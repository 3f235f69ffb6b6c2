/*
 * wide_f32_3eq.cu -- other layouts of the configurations of kern_f32_3eq.cu.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(float, CUOPO_F32, 3, 512, 1, 1, 128, 1, 1, 2.9, 4.1),
    CUOPO_W(float, CUOPO_F32, 3, 1024, 1, 1, 256, 1, 1, 3.9, 3.9),
    CUOPO_W(float, CUOPO_F32, 3, 1024, 1, 4, 192, 1, 4, 3.6, 3.7),
    CUOPO_W(float, CUOPO_F32, 3, 2048, 1, 1, 384, 1, 1, 7, 7),
    CUOPO_W(float, CUOPO_F32, 3, 2048, 1, 4, 128, 1, 1, 4, 4.3),
    CUOPO_W(float, CUOPO_F32, 3, 2048, 1, 8, 192, 1, 4, 3.6, 3.8),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 1, 2, 384, 1, 1, 9.6, 9.6),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 1, 4, 256, 1, 1, 4.5, 4.5),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 1, 16, 128, 1, 1, 3.7, 3.9),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 2, 4, 384, 1, 1, 9.6, 9.6),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 2, 8, 256, 1, 1, 5.3, 5.3),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 2, 16, 256, 1, 1, 3.8, 3.8),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 4, 8, 384, 1, 1, 11, 11),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 4, 16, 256, 1, 1, 6, 6),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 8, 16, 384, 1, 1, 11.4, 11.4),
    CUOPO_W(float, CUOPO_F32, 3, 4096, 16, 16, 384, 1, 1, 21.6, 21.6),
    /* more instances than fit one CTA per SM: in place, two per SM */
    CUOPO_K(float, CUOPO_F32, 3, 4096, 1, 1, 2, 13.9, 20.5),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 4, 1, 2, 18, 26.7),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 8, 1, 2, 21.7, 35.4),
    CUOPO_K(float, CUOPO_F32, 3, 4096, 16, 1, 2, 25, 42),
};

const KernelList wide_f32_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
