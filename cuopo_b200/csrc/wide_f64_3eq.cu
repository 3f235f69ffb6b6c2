/*
 * wide_f64_3eq.cu -- other layouts of the configurations of kern_f64_3eq.cu.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(double, CUOPO_F64, 3, 512, 1, 1, 128, 1, 1, 4.9, 7.2),
    CUOPO_W(double, CUOPO_F64, 3, 1024, 1, 1, 256, 1, 1, 7.1, 7.1),
    CUOPO_W(double, CUOPO_F64, 3, 1024, 1, 4, 128, 1, 1, 6, 6.6),
    CUOPO_W(double, CUOPO_F64, 3, 2048, 1, 4, 128, 1, 1, 8.3, 8.8),
    CUOPO_W(double, CUOPO_F64, 3, 2048, 1, 8, 128, 1, 1, 6.5, 6.8),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 1, 4, 256, 1, 1, 8.7, 8.7),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 1, 16, 128, 1, 1, 6.5, 6.6),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 2, 8, 256, 1, 1, 9.3, 9.3),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 2, 16, 256, 1, 1, 6.6, 6.6),
    CUOPO_W(double, CUOPO_F64, 3, 2048, 8, 8, 256, 1, 1, 18.6, 18.6),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 8, 16, 384, 1, 1, 20.2, 20.2),
};

const KernelList wide_f64_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
