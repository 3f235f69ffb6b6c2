/*
 * wide_f64_3eq.cu -- few-instance kernel configurations of FP64 fields, 3 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_W(double, CUOPO_F64, 3, 512, 1, 2, 256),
    CUOPO_W(double, CUOPO_F64, 3, 1024, 1, 4, 256),
    CUOPO_W(double, CUOPO_F64, 3, 2048, 1, 8, 256),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 1, 16, 256),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 2, 16, 256),
    CUOPO_W(double, CUOPO_F64, 3, 2048, 8, 8, 384),
    CUOPO_W(double, CUOPO_F64, 3, 4096, 8, 16, 384),
};

const KernelList wide_f64_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
