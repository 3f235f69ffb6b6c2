/*
 * solo_f32_2eq.cu -- FP32 fields, 2 equations: the configurations of
 * kern_f32_2eq.cu that keep two CTAs on an SM, for launches that have no more
 * than one per SM: twice the registers (nothing spilled) and one copy of the
 * field step's code (kernels of several grid sizes share instruction caches).
 * 36 instances of 2^12..2^15 take 16.4 us per slice, 21.6 with the kernels
 * of two CTAs per SM; 148 of 2^12 take 10.3 us (11.1),
 * 74 of 2^13 12.8 (13.9).
 */
#include "kernels.cuh"

namespace cuopo {

static const KernelEntry k_list[] = {
    CUOPO_KC(float, CUOPO_F32, 2, 4096, 1, 0, 1, 1, 10.3, 10.3),
    CUOPO_KC(float, CUOPO_F32, 2, 4096, 2, 0, 1, 1, 12.8, 12.8),
    CUOPO_KC(float, CUOPO_F32, 2, 4096, 4, 0, 1, 1, 13.8, 13.8),
    CUOPO_KC(float, CUOPO_F32, 2, 4096, 8, 0, 1, 1, 15.5, 15.5),
};

const KernelList solo_f32_2eq = {k_list, (int)(sizeof(k_list) / sizeof(k_list[0]))};

}  // namespace cuopo
