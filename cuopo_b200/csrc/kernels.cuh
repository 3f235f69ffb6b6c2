/*
 * kernels.cuh -- the built kernel configurations: their launch functions and
 * the registry entries.  Each kern_*.cu instantiates the configurations of
 * one precision and number of equations (separate files so that they compile
 * in parallel); solver.cu chooses among them.
 */
#pragma once
#include <cstring>

#include "cuopo.h"
#include "ssfm.cuh"

namespace cuopo {

typedef cudaError_t (*launch_fn)(const LaunchArgs &, int clusters, cudaStream_t);
typedef int (*occ_fn)(void);

template <typename R, int F, int M, int CL, int HM, int MINB>
static cudaError_t prepare_kernel()
{
    using K = Ssfm<R, F, M, CL, HM>;
    static cudaError_t st = [] {
        cudaError_t e = cudaFuncSetAttribute(ssfm_kernel<R, F, M, CL, HM, MINB>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem_bytes());
        if (e == cudaSuccess && CL > 8)
            e = cudaFuncSetAttribute(ssfm_kernel<R, F, M, CL, HM, MINB>,
                                     cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e;
    }();
    return st;
}

template <typename R, int F, int M, int CL, int HM, int MINB>
static cudaLaunchConfig_t make_config(int clusters, cudaStream_t st, cudaLaunchAttribute *attr)
{
    using K = Ssfm<R, F, M, CL, HM>;
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(clusters * CL));
    cfg.blockDim = dim3(K::T);
    cfg.dynamicSmemBytes = K::smem_bytes();
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <typename R, int F, int M, int CL, int HM, int MINB>
static cudaError_t launch_impl(const LaunchArgs &a, int clusters, cudaStream_t st)
{
    cudaError_t e = prepare_kernel<R, F, M, CL, HM, MINB>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = make_config<R, F, M, CL, HM, MINB>(clusters, st, attr);
    e = cudaLaunchKernelEx(&cfg, ssfm_kernel<R, F, M, CL, HM, MINB>, a);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

/* Clusters (of CL CTAs) of this kernel that can be resident at once (0 on error). */
template <typename R, int F, int M, int CL, int HM, int MINB>
static int occupancy_impl()
{
    if (prepare_kernel<R, F, M, CL, HM, MINB>() != cudaSuccess) return 0;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = make_config<R, F, M, CL, HM, MINB>(1, 0, attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, ssfm_kernel<R, F, M, CL, HM, MINB>, &cfg) != cudaSuccess) return 0;
    return n;
}

struct KernelEntry {
    int precision, F, M, CL;
    int home; /* 0, 1: fields in shared memory (1: in place); 2: in global memory */
    size_t smem;
    launch_fn fn;
    occ_fn occ;
};

#define CUOPO_K(R, PREC, F, M, CL, HM, MINB)                                                  \
    {PREC, F, M, CL, HM, Ssfm<R, F, M, CL, HM>::smem_bytes(), &launch_impl<R, F, M, CL, HM, MINB>, \
     &occupancy_impl<R, F, M, CL, HM, MINB>}

/* Configurations of one precision and number of equations. */
struct KernelList {
    const KernelEntry *k;
    int n;
};
extern const KernelList kern_f32_2eq, kern_f32_3eq, kern_f64_2eq, kern_f64_3eq;

}  // namespace cuopo
