/*
 * wide_f64_2eq.cu -- other layouts of the configurations of kern_f64_2eq.cu.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(double, CUOPO_F64, 2, 512, 1, 1, 128, 1, 1, 4.9, 7.1),
    CUOPO_W(double, CUOPO_F64, 2, 512, 1, 2, 128, 1, 1, 4.6, 5.6),
    CUOPO_W(double, CUOPO_F64, 2, 1024, 1, 1, 256, 1, 1, 6.5, 6.5),
    CUOPO_W(double, CUOPO_F64, 2, 1024, 1, 4, 128, 1, 1, 5.2, 5.6),
    CUOPO_W(double, CUOPO_F64, 2, 2048, 1, 4, 128, 1, 1, 7.8, 8.5),
    CUOPO_W(double, CUOPO_F64, 2, 2048, 1, 8, 128, 1, 1, 5.7, 5.9),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 1, 2, 256, 1, 1, 13.8, 13.8),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 1, 4, 256, 1, 1, 8, 8),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 1, 16, 128, 1, 1, 5.8, 5.9),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 2, 4, 256, 1, 1, 14.4, 14.4),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 2, 8, 256, 1, 1, 8.7, 8.7),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 2, 16, 256, 1, 1, 6.4, 6.4),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 4, 8, 256, 1, 1, 14.8, 14.8),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 4, 16, 256, 1, 1, 9.1, 9.1),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 8, 16, 256, 1, 1, 16.2, 16.2),
};

const KernelList wide_f64_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
