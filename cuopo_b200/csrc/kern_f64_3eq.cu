/*
 * kern_f64_3eq.cu -- kernel configurations of FP64 fields, 3 equations.
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_K(double, CUOPO_F64, 3, 512, 1, 0, 1, 11.1, 16.9),
    CUOPO_K(double, CUOPO_F64, 3, 1024, 1, 0, 1, 11.5, 17.4),
    CUOPO_K(double, CUOPO_F64, 3, 2048, 1, 0, 1, 12.5, 12.5),
    CUOPO_K(double, CUOPO_F64, 3, 4096, 1, 1, 1, 22.2, 22.2),
    CUOPO_K(double, CUOPO_F64, 3, 4096, 2, 1, 1, 27.2, 27.2),
    CUOPO_K(double, CUOPO_F64, 3, 2048, 8, 0, 1, 22, 22),
    CUOPO_K(double, CUOPO_F64, 3, 4096, 8, 1, 1, 37.9, 37.9),
    CUOPO_K(double, CUOPO_F64, 3, 4096, 16, 1, 1, 0, 0),
    /* 2^17 FP64 points of 3 fields (6 MiB) exceed the shared memory of a
     * 16-CTA cluster: the fields stay in global memory (L2) */
    CUOPO_K(double, CUOPO_F64, 3, 8192, 16, 2, 1, 0, 0),
};

const KernelList kern_f64_3eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
