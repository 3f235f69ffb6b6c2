/*
 * wide_f64_2eq.cu -- few-instance kernel configurations of FP64 fields, 2 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(double, CUOPO_F64, 2, 512, 1, 2, 256),
    CUOPO_W(double, CUOPO_F64, 2, 1024, 1, 4, 256),
    CUOPO_W(double, CUOPO_F64, 2, 2048, 1, 8, 256),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 1, 16, 256),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 2, 16, 256),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 4, 16, 256),
    CUOPO_W(double, CUOPO_F64, 2, 4096, 8, 16, 256),
};

const KernelList wide_f64_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
