/*
 * kern_f64_2eq.cu -- kernel configurations of FP64 fields, 2 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(double, CUOPO_F64, 2, 512, 1, 0, 1, 10.9, 17.1),
    CUOPO_K(double, CUOPO_F64, 2, 1024, 1, 0, 1, 11, 17.2),
    CUOPO_K(double, CUOPO_F64, 2, 2048, 1, 0, 1, 11.9, 17.6),
    CUOPO_K(double, CUOPO_F64, 2, 4096, 1, 0, 1, 19.6, 19.6),
    CUOPO_K(double, CUOPO_F64, 2, 4096, 2, 0, 1, 22.4, 22.4),
    CUOPO_K(double, CUOPO_F64, 2, 4096, 4, 0, 1, 24.2, 24.2),
    CUOPO_K(double, CUOPO_F64, 2, 4096, 8, 0, 1, 29.2, 29.2),
    CUOPO_K(double, CUOPO_F64, 2, 4096, 16, 0, 1, 0, 0),
};

const KernelList kern_f64_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
