/*
 * kernels.cuh -- the built kernel configurations: their launch functions and
 * the registry entries.  Each kern_*.cu and solo_*.cu (ssfm_kernel) and wide_*.cu
 * (wide_kernel) instantiates the configurations of one precision and number
 * of equations (separate files so that they compile in parallel); solver.cu
 * chooses among them.
 */
#pragma once
#include <cstring>

#include "cuopo.h"
#include "wide.cuh"

namespace cuopo {

typedef cudaError_t (*launch_fn)(const LaunchArgs &, int clusters, bool spread, cudaStream_t);
typedef int (*occ_fn)(void);

/* Dynamic shared memory that keeps any two CTAs off one SM (227 KB each). */
constexpr size_t SPREAD_SMEM = 116 * 1024;

/* Launches of one kernel: CLUSTER CTAs per instance, THREADS per CTA.
 * spread: one CTA per SM. */
template <void (*KERNEL)(LaunchArgs), int CLUSTER, int THREADS, size_t SMEM>
struct Launcher {
    static cudaError_t prepare()
    {
        static cudaError_t st = [] {
            cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)(SMEM > SPREAD_SMEM ? SMEM : SPREAD_SMEM));
            if (e == cudaSuccess && CLUSTER > 8)
                e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            return e;
        }();
        return st;
    }

    static cudaLaunchConfig_t config(int clusters, cudaStream_t st, cudaLaunchAttribute *attr)
    {
        cudaLaunchConfig_t cfg;
        std::memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3((unsigned)(clusters * CLUSTER));
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = SMEM;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CLUSTER;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cfg;
    }

    static cudaError_t launch(const LaunchArgs &a, int clusters, bool spread, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t cfg = config(clusters, st, attr);
        if (spread && SMEM < SPREAD_SMEM) cfg.dynamicSmemBytes = SPREAD_SMEM;
        e = cudaLaunchKernelEx(&cfg, KERNEL, a);
        if (e != cudaSuccess) return e;
        return cudaGetLastError();
    }

    /* Clusters that can be resident at once (0 on error). */
    static int occupancy()
    {
        static const int clusters = [] {
            cudaLaunchAttribute attr[1];
            cudaLaunchConfig_t cfg = config(1, 0, attr);
            int n = 0;
            if (prepare() != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, KERNEL, &cfg) != cudaSuccess) n = 0;
            return n;
        }();
        return clusters;
    }
};

struct KernelEntry {
    int precision, F, M, CL;
    int home;           /* 0, 1: fields in shared memory (1: in place); 2: in global memory */
    int ctas, threads;  /* per instance, per CTA */
    int wide;           /* wide_kernel: its order of the frequency tables (freq_slot) */
    float us1, us_full; /* measured time per slice [us] with at most one CTA per SM, and with every
                           resident cluster busy (B200, 1965 MHz); 0: not compared */
    size_t smem;
    launch_fn fn;
    occ_fn occ;
};

#define CUOPO_K(R, PREC, F, M, CL, HM, MINB, US1, USF)                                                         \
    CUOPO_KC(R, PREC, F, M, CL, HM, MINB, field_copies<R>(F), US1, USF)
#define CUOPO_KC(R, PREC, F, M, CL, HM, MINB, COPIES, US1, USF)                                                \
    {PREC, F, M, CL, HM, CL, M / 16, 0, US1, USF, Ssfm<R, F, M, CL, HM>::smem_bytes(),                          \
     &Launcher<&ssfm_kernel<R, F, M, CL, HM, MINB, COPIES>, CL, M / 16,                                         \
               Ssfm<R, F, M, CL, HM>::smem_bytes()>::launch,                                                    \
     &Launcher<&ssfm_kernel<R, F, M, CL, HM, MINB, COPIES>, CL, M / 16,                                         \
               Ssfm<R, F, M, CL, HM>::smem_bytes()>::occupancy}

/* The same arithmetic (M, CL) spread over P CTAs of NTHR threads, at least
 * MINB on an SM, Q threads per 16-point transform (wide.cuh). */
#define CUOPO_W(R, PREC, F, M, CL, P, NTHR, MINB, Q, US1, USF)                                                 \
    {PREC, F, M, CL, 0, P, NTHR, 1, US1, USF, Wide<R, F, M, CL, P, NTHR, MINB, Q>::smem_bytes(),                \
     &Launcher<&wide_kernel<R, F, M, CL, P, NTHR, MINB, Q>, P, NTHR,                                            \
               Wide<R, F, M, CL, P, NTHR, MINB, Q>::smem_bytes()>::launch,                                      \
     &Launcher<&wide_kernel<R, F, M, CL, P, NTHR, MINB, Q>, P, NTHR,                                            \
               Wide<R, F, M, CL, P, NTHR, MINB, Q>::smem_bytes()>::occupancy}

/* Configurations of one precision and number of equations. */
struct KernelList {
    const KernelEntry *k;
    int n;
};
extern const KernelList kern_f32_2eq, kern_f32_3eq, kern_f64_2eq, kern_f64_3eq;
extern const KernelList solo_f32_2eq;
extern const KernelList wide_f32_2eq, wide_f32_3eq, wide_f64_2eq, wide_f64_3eq;

}  // namespace cuopo
