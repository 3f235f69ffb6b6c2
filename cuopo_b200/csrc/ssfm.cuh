/*
 * ssfm.cuh -- the fused SSFM round-trip kernel.
 *
 * One launch runs whole crystal passes and cavity round trips of the
 * reference loop (src/cuOPO.cu:474-610) with every field resident in shared
 * memory, for one instance per CTA (CL = 1) or per thread-block cluster of
 * CL CTAs (grids up to CL x 8192 points):
 *
 *   per round trip:  pump injection (cuOPO.cu:478-486, functions.cuh:191-213)
 *     per slice s:   RK4 half step at z_s (cwes2.cuh:147-166)
 *                    for each field: T->W transform (CUFFT_INVERSE), x D(w)/N
 *                    (LinearOperator + CUFFTscale, cwes2.cuh:103-121,
 *                    functions.cuh:126-135), W->T transform (CUFFT_FORWARD)
 *                    RK4 half step at z_s again (cwes2.cuh:188-207, quirk Q2)
 *     EOM (functions.cuh:242-253), GDD/TOD (cuOPO.cu:521-553), AddPhase
 *     (functions.cuh:139-152), SaveRoundTrip (functions.cuh:217-238), and
 *     the signal power for the convergence rule.
 *
 * Cluster decomposition (N = CL * M): CTA c holds time block n = n1 + M c.
 * The T->W transform is a radix-CL "cross" stage over the CTAs,
 *   y_k2[n1] = W_N^{n1 k2} sum_n2 x[n1 + M n2] W_CL^{n2 k2}   (stored on CTA k2),
 * followed by a local M-point transform on CTA k2 giving X[k2 + CL k1]; the
 * W->T transform runs the same two steps backwards.  Between the local W->T
 * transform of slice s and the local T->W transform of slice s+1 the
 * inverse cross stage, both RK4 half steps and the forward cross stage are
 * one element-wise pass over distributed shared memory, so each slice costs
 * one exchange between the CTAs and two cluster barriers.  The fields live
 * in the y domain between slices; the time domain exists only inside that
 * pass (and at round-trip ends).  With CL = 1 the cross stages are
 * identities and no barrier is needed around the element-wise passes.
 *
 * Quirks kept: RK4 stages use aux = A + s k without the step (Q1); both
 * half steps of a slice use the same z (Q2); in the 3-equation model all
 * stages read the unperturbed fields (Q3), so the half step reduces to
 * A += c(z) * P(A) with one coefficient per field and slice.
 */
#pragma once
#include <cooperative_groups.h>

#include "fft.cuh"

namespace cuopo {

/* Per-plan device tables (type-erased; element type is cpx<R>).  Tables
 * indexed by frequency are stored per CTA: entry [k2][k1] is frequency
 * index k2 + CL k1. */
struct Tables {
    const void *disp;   /* [F][CL][M]: slice dispersion x attenuation / N */
    const void *rk;     /* [n_z + 1][4]: RK4 half steps, see RkRow */
    const void *eom;    /* [N]: exp(i m sin(2 pi fpm T)) or NULL */
    const float *w;     /* [CL][M]: angular frequency grid (reference float values) */
    const void *twN;    /* [CL - 1][M]: W_N^{n1 c} at [c - 1][n1] (cross-stage twiddles; CL > 1): the lanes of a
                         * warp (consecutive n1) read one run per c (indexed by n1 c they read up to 14 lines) */
    const double2 *frame_u; /* [NFRAME]: random frame angles (u_s, u_i) in turns, |u| < 1/8 */
    const void *frame_c;    /* [NFRAME][3]: rotation (tan, sin) for pump, signal, idler */
    double h6;          /* (dz/2)/6 */
    double kp, ks;      /* 2 eqs: couplings */
    double g_last;      /* pump frame of the last slice [turns] */
    double inv_n;       /* 1/N */
};

/* One OPO instance (one set of fields and cavity settings). */
struct Instance {
    void *Ap, *As, *Ai;         /* device fields, n_t values each */
    const void *pump;           /* CW: n_t values or NULL (constant ap0); NS: window */
    double ap0;                 /* constant CW pump amplitude when pump == NULL */
    int n_rt_total;             /* NRT of the NS pump window (ReadPump) */
    int rt_begin, rt_count;
    void *sv_p, *sv_s, *sv_i;   /* SaveRoundTrip buffers (may be NULL) */
    int save_first, save_count;
    double *ps_hist;            /* per-rt signal power (may be NULL) */
    double tol;                 /* convergence tolerance (<= 0: off) */
    int *rt_done;               /* number of round trips run (may be NULL) */
    double phase_s[2];          /* sqrt(Rs) exp(i pi delta) */
    double phase_i[2];          /* sqrt(Ri) exp(i pi delta) */
    double gdd;                 /* intracavity GDD [ps^2]; 0 = off */
    double tod_s, tod_i;        /* TOD compensation [ps^3] */
    int use_tod_s, use_tod_i;
    int patience;               /* consecutive rts below tol to stop (>= 1) */
    double *ps_out;             /* final signal power (may be NULL) */
    int *flag_out;              /* 1 converged, 0 max rts reached, 5 non-finite (may be NULL) */
    /* resumable state of a batch instance (all NULL for single launches):
     * round trips run so far, last signal power, calm-rt counter and flag
     * (0 running, 1 converged, 2 round-trip limit reached, 5 non-finite) */
    int *st_rt;
    double *st_ps;
    int *st_calm;
    int *st_flag;
    /* the instance's own physics tables (batches whose instances differ in
     * crystal, wavelengths, length or modulator); NULL disp: the launch's */
    const void *disp, *rk, *eom;
    const float *w;
    double h6, kp, ks, g_last;
};

struct LaunchArgs {
    Tables tab;
    Instance single;            /* used when inst == NULL */
    const Instance *inst;       /* batch of instances, or NULL */
    int n_inst;
    int *queue;                 /* work-queue counter for persistent batches */
    int n_z;
    int regime;                 /* CUOPO_CW / CUOPO_NS */
    int pass_only;              /* 1: one crystal pass, no cavity map */
    int use_eom, eom_idler;
    int *status;                /* first error code (atomicCAS from 0) */
    int hold;                   /* test hook: exchanges into the first CTA of an instance never complete, so
                                   its bounded waits run out (wide_kernel) */
    /* batch launches: continue each running instance by up to `chunk` round
     * trips, stopping at max_rt; convergence tolerance and patience */
    int chunk, max_rt, patience;
    double tol;
};

enum { ST_OK = 0, ST_CONVERGED = 1, ST_LIMIT = 2, ST_TIMEOUT = 4, ST_NONFINITE = 5 };

/* Random frame rotations.  The coupled-wave equations are invariant under
 * (Ap, As, Ai) -> (Ap e^{i(a+b)}, As e^{ia}, Ai e^{ib}) (and Ap e^{2ia} in the
 * degenerate 2-equation model), and the linear steps commute with it.  Each
 * slice the kernel moves the fields to a new frame drawn from a fixed table
 * and returns them to the laboratory frame before the cavity map; the
 * rounding errors of the float transforms then have random phase relative
 * to the field, so they do not add up coherently over the ~10^5 slices of a
 * run.  Entry of slice s of round trip rt: frame_index(rt, s). */
enum { NFRAME = 1024 };

__host__ __device__ __forceinline__ int frame_index(int rt, int s)
{
    unsigned long long z = ((unsigned long long)(unsigned)rt << 32) ^ (unsigned)s ^ 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (int)(z & (NFRAME - 1));
}

template <typename C>
__device__ __forceinline__ C ldc(const void *p, long i)
{
    return __ldg(reinterpret_cast<const C *>(p) + i);
}

/*
 * RK4 half steps in the pump frame.  The stage coefficients of slice s are
 * i kp e^{+i dk z_j} and i ks e^{-i dk z_j} (z_j = z, z+dz/4, z+dz/2), so with
 * the pump turned by g_s = -dk (z_s + dz/4) the two middle stages have no
 * phase at all and the outer two e1 = e^{-i dk dz/4} and e2 = e^{i dk dz/4}
 * or their conjugates; kp, ks go into the scalars of the updates.  That is
 * 76 multiply-adds per point and half step against 96 with a complex
 * coefficient per stage, for one more rotation of the pump per slice (3).
 * The 3-equation half step (one coefficient h6 i kappa_f (E(z) +
 * 4 E(z+dz/4) + E(z+dz/2)) per field, E conjugate for the pump) becomes
 * purely imaginary in the frame of that sum's phase: 18 against 30.  The
 * kernel's other steps commute with a constant turn of the pump.
 *
 * Row s < n_z of the table, 4 complex entries:
 *   2 eqs: e1, e2;  3 eqs: (c_p, c_s), (c_i, 0) with A_f += i c_f P_f
 *   (tan(phi/2), sin(phi)) and (m, 0): the turn of the pump from the frame of
 *   slice s to that of slice s+1 as m quarter turns and a rotation phi;
 * row n_z holds the turn from the laboratory frame into slice 0's.
 */
template <typename R>
struct RkConst {
    R hp, hs, fp, fs, gp, gs;   /* kappa/2, kappa, h6 kappa */
};

/* 2 equations: cwes2.cuh:30-87. */
template <typename C, typename R>
__device__ __forceinline__ void rk4_half2(C &Ap, C &As, C e1, C e2, const RkConst<R> &k)
{
    const C g1p = cmul(cisq(As), e1);
    const C g1s = cmulc(cimulc(Ap, As), e1);
    C ap = caxpy(Ap, k.hp, g1p), as = caxpy(As, k.hs, g1s);
    const C g2p = cisq(as);
    const C g2s = cimulc(ap, as);
    ap = caxpy(Ap, k.hp, g2p);
    as = caxpy(As, k.hs, g2s);
    const C g3p = cisq(as);
    const C g3s = cimulc(ap, as);
    ap = caxpy(Ap, k.fp, g3p);
    as = caxpy(As, k.fs, g3s);
    const C g4p = cmul(cisq(as), e2);
    const C g4s = cmulc(cimulc(ap, as), e2);
    Ap = caxpy(Ap, k.gp, caxpy(cadd(g1p, g4p), (R)2, cadd(g2p, g3p)));
    As = caxpy(As, k.gs, caxpy(cadd(g1s, g4s), (R)2, cadd(g2s, g3s)));
}

/* 3 equations: cwes3.cuh:30-90 with Q3, P = (As Ai, Ap conj(Ai), Ap conj(As)). */
template <typename C>
__device__ __forceinline__ void rk4_half3(C &Ap, C &As, C &Ai, C c0, C c1)
{
    const C Pp = cimul(As, Ai);
    const C Ps = cimulc(Ap, Ai);
    const C Pi = cimulc(Ap, As);
    Ap = caxpy(Ap, c0.x, Pp);
    As = caxpy(As, c0.y, Ps);
    Ai = caxpy(Ai, c1.x, Pi);
}

namespace cg = cooperative_groups;

/* Where the fields live during a launch (HM):
 *   0  shared memory: home[F][M] and a scratch[M] for the local transforms
 *   1  shared memory, in place: home[F][M], the local transforms exchange
 *      through the field's own home
 *   2  global memory: the caller's field buffers, L2-resident between
 *      passes, with one shared scratch[M] for the local transforms; for grids
 *      whose fields exceed a cluster's shared memory (3 FP64 fields of 2^17
 *      points are 6 MiB, a 16-CTA cluster has 3.6 MB).  Every access to
 *      the fields goes to L2 (ld/st .cg), ordered by the cluster barriers.
 * COPIES: copies of a field's dispersion step in the code (Engine::dispersion). */
template <typename R>
constexpr int field_copies(int F) { return sizeof(R) == 4 && F == 2 ? F : 1; }

template <typename R, int F, int M, int CL, int HM, int COPIES = field_copies<R>(F)>
struct Ssfm {
    static constexpr bool GH = (HM == 2);
    static constexpr bool INPLACE = (HM != 0); /* one exchange buffer per local transform */
    using C = cpx<R>;
    using SP = StagePlan<M>;
    static constexpr int T = SP::T;
    static constexpr int P = SP::P;
    static constexpr int N = M * CL;
    static constexpr int J = 16 / CL;  /* n1 values per thread in a cross stage */
    static constexpr int NCO = 4;      /* entries of a row of the RK4 table */
    static constexpr unsigned ALL = (1u << F) - 1u;
    static_assert(CL == 1 || CL == 2 || CL == 4 || CL == 8 || CL == 16, "cluster size must be 1..16, power of 2");

    /* Shared memory: home[F][M] (+ scratch[M]) complex values, or scratch[M]
     * alone (HM = 2), then the twiddle table of the middle FFT stages. */
    static constexpr size_t field_elems() { return GH ? (size_t)M : (size_t)M * (F + (INPLACE ? 0 : 1)); }
    static constexpr size_t smem_bytes() { return sizeof(C) * (field_elems() + TwTable<M>::size()); }

    /* Element-wise work of one cross stage (uniform over the cluster). */
    struct Ops {
        int inject;         /* pump injection */
        long poff;          /* NS pump window offset of this round trip */
        const C *rk0, *rk1; /* rows of the RK4 half steps to apply (NULL: none) */
        const C *turn;      /* row whose turn of the pump comes between the two (NULL: none) */
        int frame;          /* entry of the frame table to move to (-1: none) */
        int eom;            /* intracavity phase modulator */
        int rotate;         /* frame rotation: 1 the shear rotations rf[f], 2 quarter turns rq[f] first */
        C rf[3];
        int rq[3];
        int addphase;       /* AddPhase on the resonant fields */
        double2 ph_s, ph_i;
        int save;           /* SaveRoundTrip into slot */
        size_t slot;
        int power;          /* accumulate |As|^2 */
    };

    /* Move to the frame of a table entry (rotation by 2 pi u per field, built
     * from the shears fc); th accumulates each field's frame angle in turns
     * (the pump's starts at the RK4 frame of the last slice). */
    static __device__ __forceinline__ void frame_step(Ops &op, const C *fc, double2 u, double (&th)[3])
    {
        op.rotate = 1;
#pragma unroll
        for (int f = 0; f < 3; f++) op.rf[f] = fc[f];
        th[1] += u.x;
        th[2] += u.y;
        th[0] += (F == 2) ? 2.0 * u.x : u.x + u.y;
    }

    /* Back to the laboratory frame: rotation by -th = quarter turns plus a
     * residual of at most 1/8 turn, formed in FP64. */
    static __device__ __forceinline__ void frame_back(Ops &op, const double (&th)[3])
    {
        op.rotate = 2;
#pragma unroll
        for (int f = 0; f < 3; f++) {
            const double back = -th[f];
            const double qt = rint(4.0 * back);
            const double res = back - 0.25 * qt; /* turns, |res| <= 1/8 */
            double sh, ch, sn, cs;
            sincospi(res, &sh, &ch);
            sincospi(2.0 * res, &sn, &cs);
            op.rq[f] = ((int)fmod(qt, 4.0) + 4) & 3;
            op.rf[f] = mk<C>((R)(sh / ch), (R)sn);
        }
    }

    /* Round-trip limit of a batch instance: the launch's, and for a
     * nanosecond instance also the end of its pump window. */
    static __device__ __forceinline__ int rt_limit(const LaunchArgs &a, const Instance &I)
    {
        return (a.regime == 1 && I.n_rt_total > 0) ? min(a.max_rt, I.n_rt_total) : a.max_rt;
    }

    /* Cluster barrier (release / acquire).  Every call site is reached by
     * all threads of the cluster with uniform control flow, so the
     * warp-aligned form applies; it runs batches of 2^15-point instances
     * 1.4 % faster than the generic form (4.5 % for one instance alone). */
    static __device__ __forceinline__ void csync()
    {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    static __device__ __forceinline__ void xsync()
    {
        if constexpr (GH) {
            /* the cross passes write other CTAs' positions of global memory */
            __threadfence();
            if constexpr (CL > 1) csync();
            else __syncthreads();
        } else if constexpr (CL > 1) {
            csync();
        }
    }

    static __device__ __forceinline__ void bar()
    {
        if constexpr (CL > 1) csync();
        else __syncthreads();
    }

    template <typename X>
    static __device__ __forceinline__ X *peer(X *p, int rank)
    {
        if constexpr (CL == 1) return p;
        else return cg::this_cluster().map_shared_rank(p, rank);
    }

    static __device__ __forceinline__ C mul_fp64(C a, double2 f)
    {
        const double re = rfma((double)a.x, f.x, -rmul((double)a.y, f.y));
        const double im = rfma((double)a.x, f.y, rmul((double)a.y, f.x));
        return mk<C>((R)re, (R)im);
    }

    /* Table entries of one cross pass, loaded once (through a pointer they
     * would be reloaded for every point: the shared-memory stores between
     * points may alias it for the compiler). */
    struct Coef {
        C a0, a1, b0, b1;   /* the two half steps */
        C turn;             /* turn of the pump between them: rotation, quarter turns */
        int turn_q;
        RkConst<R> k;
    };

    /* The coefficients of the next pass in shared memory: the last warp loads
     * them before the dispersion step (one entry per lane, in flight
     * meanwhile) and writes them before a barrier in it, so that no pass
     * waits for them. */
    struct Staged {
        C c[9];      /* rk0: 2, turn: 2, rk1: 2, frame rotations: 3 */
        double2 u;   /* frame angles */
    };

    struct Stager {
        C pf;
        double2 pf_u;

        /* lane l >= 0 of the last warp */
        __device__ __forceinline__ void load(int l, const Ops &op, const Tables &tab)
        {
            const C *src = nullptr;
            pf = mk<C>((R)0, (R)0);
            if (l < 0) return;
            if (l < 2) src = op.rk0 ? op.rk0 + l : nullptr;
            else if (l < 4) src = op.turn ? op.turn + l : nullptr;
            else if (l < 6) src = op.rk1 ? op.rk1 + (l - 4) : nullptr;
            else if (l < 9 && op.frame >= 0) src = reinterpret_cast<const C *>(tab.frame_c) + 3 * op.frame + (l - 6);
            if (src) pf = __ldg(src);
            if (l == 9 && op.frame >= 0) pf_u = tab.frame_u[op.frame];
        }

        __device__ __forceinline__ void write(int l, Staged *s) const
        {
            if (l >= 0 && l < 9) s->c[l] = pf;
            if (l == 9) s->u = pf_u;
        }
    };

    static __device__ __forceinline__ Coef coef(const Staged *s, const RkConst<R> &k)
    {
        Coef c;
        c.k = k;
        c.a0 = s->c[0];
        c.a1 = s->c[1];
        c.turn = s->c[2];
        c.turn_q = (int)s->c[3].x;
        c.b0 = s->c[4];
        c.b1 = s->c[5];
        return c;
    }

    static __device__ __forceinline__ void half_step(C (&A)[3], C c0, C c1, const RkConst<R> &k)
    {
        if constexpr (F == 2) rk4_half2(A[0], A[1], c0, c1, k);
        else rk4_half3(A[0], A[1], A[2], c0, c1);
    }

    static __device__ __forceinline__ void pointwise(C (&A)[3], int n, const Ops &op, const Coef &co,
                                                     const Instance &I, const Tables &tab, int eom_idler, double &acc)
    {
        if (op.inject) A[0] = I.pump ? ldc<C>(I.pump, op.poff + n) : mk<C>((R)I.ap0, (R)0);
        if (op.rk0) half_step(A, co.a0, co.a1, co.k);
        if (op.turn) {
            if (co.turn_q) A[0] = iq_rt(A[0], co.turn_q);
            A[0] = shear_rot(A[0], co.turn.x, co.turn.y);
        }
        if (op.rk1) half_step(A, co.b0, co.b1, co.k);
        if (op.eom) {
            const C ef = ldc<C>(tab.eom, n);
            A[1] = cmul(A[1], ef);
            if (F == 3 && eom_idler) A[F - 1] = cmul(A[F - 1], ef);
        }
        if (op.rotate) {
            if (op.rotate == 2) {
#pragma unroll
                for (int f = 0; f < F; f++) A[f] = iq_rt(A[f], op.rq[f]);
            }
#pragma unroll
            for (int f = 0; f < F; f++) A[f] = shear_rot(A[f], op.rf[f].x, op.rf[f].y);
        }
        if (op.addphase) {
            /* in FP64 so that sqrt(R) exp(i pi delta) carries no float rounding
             * bias into the round-trip gain */
            A[1] = mul_fp64(A[1], op.ph_s);
            if constexpr (F == 3) A[2] = mul_fp64(A[2], op.ph_i);
        }
        if (op.save) {
            C *sv[3] = {reinterpret_cast<C *>(I.sv_p), reinterpret_cast<C *>(I.sv_s),
                        reinterpret_cast<C *>(I.sv_i)};
#pragma unroll
            for (int f = 0; f < F; f++)
                if (sv[f]) sv[f][op.slot + n] = A[f];
        }
        if (op.power) acc += cabs2d(A[1]);
    }

    /* The radix-CL stages of one field at position n1: the inverse one (y ->
     * time) and the forward one, with the cross-stage twiddles W_N^{n1 c}:
     * quarter turn and residual rotation (tan, sin) from the table. */
    static __device__ __forceinline__ void cross_inv(C (&v)[CL], int n1, const C *__restrict__ twN)
    {
#pragma unroll
        for (int c = 1; c < CL; c++) {
            const int q = n1 * c;
            const C w = __ldg(twN + (c - 1) * M + n1);
            v[c] = shear_rot(iq_rt(v[c], (-((4 * q + N / 2) / N)) & 3), -w.x, -w.y);
        }
        dft<-1, CL>(v);
    }

    static __device__ __forceinline__ void cross_fwd(C (&v)[CL], int n1, const C *__restrict__ twN)
    {
        dft<+1, CL>(v);
#pragma unroll
        for (int c = 1; c < CL; c++) {
            const int q = n1 * c;
            const C w = __ldg(twN + (c - 1) * M + n1);
            v[c] = shear_rot(iq_rt(v[c], ((4 * q + N / 2) / N) & 3), w.x, w.y);
        }
    }

    /* The radix-CL stage of one field at the owned position n1 (S = -1: the
     * inverse cross stage, y -> time; S = +1: the forward one), on global
     * memory. */
    template <int S>
    static __device__ __forceinline__ void cross_field(C *g, const C *__restrict__ twN, int n1)
    {
        C v[CL];
#pragma unroll
        for (int c = 0; c < CL; c++) v[c] = __ldcg(g + (size_t)c * M + n1);
        if constexpr (S < 0) cross_inv(v, n1, twN);
        else cross_fwd(v, n1, twN);
#pragma unroll
        for (int c = 0; c < CL; c++) __stcg(g + (size_t)c * M + n1, v[c]);
    }

    /* The element-wise pass of `cross` with the fields in global memory
     * (HM = 2): the same arithmetic in the same order, but one field's
     * radix-CL stage at a time, the intermediate values going through L2 (CL
     * values of 3 FP64 fields would not fit in registers).  Thread t still
     * reads and writes only its own positions, so these steps need no
     * barrier between them. */
    static __device__ __forceinline__ void cross_global(C *const (&gf)[3], unsigned in_y, unsigned out_y,
                                                        const Ops &op, const Instance &I, const Tables &tab,
                                                        const Coef &co, int eom_idler, double &acc, int t, int rank)
    {
        const C *__restrict__ twN = reinterpret_cast<const C *>(tab.twN);
#pragma unroll 1
        for (int j = 0; j < J; j++) {
            const int n1 = rank * (M / CL) + t + j * T;
            if constexpr (CL > 1) {
#pragma unroll 1
                for (int f = 0; f < F; f++)
                    if ((in_y >> f) & 1u) cross_field<-1>(gf[f], twN, n1);
            }
#pragma unroll 2
            for (int c = 0; c < CL; c++) {
                C A[3];
#pragma unroll
                for (int f = 0; f < F; f++) A[f] = __ldcg(gf[f] + (size_t)c * M + n1);
                pointwise(A, n1 + M * c, op, co, I, tab, eom_idler, acc);
#pragma unroll
                for (int f = 0; f < F; f++) __stcg(gf[f] + (size_t)c * M + n1, A[f]);
            }
            if constexpr (CL > 1) {
#pragma unroll 1
                for (int f = 0; f < F; f++)
                    if ((out_y >> f) & 1u) cross_field<+1>(gf[f], twN, n1);
            }
        }
    }

    /* One element-wise pass over the cluster.  Fields with their bit set in
     * in_y are read in the y domain (inverse cross stage applied), the
     * others as time values; out_y likewise for the write-back.  Thread t
     * of CTA `rank` owns positions n1 = rank M/CL + t + j T, j < J, in every
     * CTA's home; it reads and writes only those. */
    static __device__ __forceinline__ void cross(C *home, C *const (&gf)[3], unsigned in_y, unsigned out_y,
                                                 const Ops &op, const Instance &I, const Tables &tab,
                                                 const Coef &co, int eom_idler, double &acc, int t, int rank)
    {
        if constexpr (GH) {
            cross_global(gf, in_y, out_y, op, I, tab, co, eom_idler, acc, t, rank);
            return;
        }
        const C *__restrict__ twN = reinterpret_cast<const C *>(tab.twN);
#pragma unroll 1
        for (int j = 0; j < J; j++) {
            const int n1 = rank * (M / CL) + t + j * T;
            const int sm = swz<C>(n1);
            C v[3][CL];
#pragma unroll
            for (int c = 0; c < CL; c++) {
                const C *src = peer(home, c);
#pragma unroll
                for (int f = 0; f < F; f++) v[f][c] = src[f * M + sm];
            }
            /* cross-stage twiddles W_N^{n1 c}: quarter turn m and the residual
             * rotation (tan, sin) from the table */
            if constexpr (CL > 1) {
#pragma unroll
                for (int f = 0; f < F; f++) {
                    if ((in_y >> f) & 1u) cross_inv(v[f], n1, twN);
                }
            }
#pragma unroll
            for (int c = 0; c < CL; c++) {
                C A[3];
#pragma unroll
                for (int f = 0; f < F; f++) A[f] = v[f][c];
                pointwise(A, n1 + M * c, op, co, I, tab, eom_idler, acc);
#pragma unroll
                for (int f = 0; f < F; f++) v[f][c] = A[f];
            }
            if constexpr (CL > 1) {
#pragma unroll
                for (int f = 0; f < F; f++) {
                    if ((out_y >> f) & 1u) cross_fwd(v[f], n1, twN);
                }
            }
#pragma unroll
            for (int c = 0; c < CL; c++) {
                C *dst = peer(home, c);
#pragma unroll
                for (int f = 0; f < F; f++) dst[f * M + sm] = v[f][c];
            }
        }
    }

    /* reg[e] times the GDD/TOD factor of frequency w[e stride] and 1/N
     * (functions.cuh:156-186, formed in FP64). */
    template <int NV>
    static __device__ __forceinline__ void gdd_factor(C (&reg)[NV], const float *__restrict__ w, int stride, double gdd,
                                                      double tod, int use_tod, R s_n)
    {
#pragma unroll 4
        for (int e = 0; e < NV; e++) {
            const double wk = (double)__ldg(w + e * stride);
            const double ph = use_tod ? 0.5 * wk * rfma(wk, gdd, rmul(wk * wk, tod) / 3.0) : 0.5 * wk * wk * gdd;
            double sn, cs;
            sincos(ph, &sn, &cs);
            /* cos(ph) - 1 = -2 sin^2(ph/2), exact for small ph */
            const double sh = sin(0.5 * ph);
            reg[e] = caddmul(cscale(reg[e], s_n), mk<C>((R)(-2.0 * sh * sh), (R)sn));
        }
    }

    /* Local T->W, multiply by a table row (or the GDD factor), local W->T. */
    template <int MODE> /* 0: table row, 1: GDD/TOD factor formed in FP64 */
    static __device__ __forceinline__ void spectral(C *home, C *scratch, const C *__restrict__ row,
                                                    const float *__restrict__ w, double gdd, double tod,
                                                    int use_tod, double inv_n, const StageTwiddles<M, C> &tw,
                                                    int t)
    {
        C reg[16];
        if constexpr (GH) {
            /* home: this CTA's M points of the field in global memory */
#pragma unroll
            for (int e = 0; e < 16; e++) reg[e] = __ldcg(home + t + e * T);
        } else {
            load_own<M>(home, reg, t);
        }
        C *bufA = GH ? scratch : (INPLACE ? home : scratch);
        C *bufB = GH ? scratch : home;
        C d[16];
        local_transform<+1, M, 0, INPLACE>(reg, bufA, bufB, tw, t, [&]() {
            if constexpr (MODE == 0) {
#pragma unroll
                for (int e = 0; e < 16; e++) d[e] = ld_now(row + t + e * T);
            }
        });
        /* the factor F = 1 + d is applied as (A + A d) / N (1/N is exact) */
        const R s_n = (R)inv_n;
        if constexpr (MODE == 0) {
#pragma unroll
            for (int e = 0; e < 16; e++) reg[e] = caddmul(cscale(reg[e], s_n), d[e]);
        } else {
            gdd_factor(reg, w + t, T, gdd, tod, use_tod, s_n);
        }
        local_transform<-1, M, P - 1, INPLACE>(reg, bufA, bufB, tw, t);
        if constexpr (GH) {
#pragma unroll
            for (int e = 0; e < 16; e++) __stcg(home + t + e * T, reg[e]);
        } else {
            store_own<M>(home, reg, t);
        }
    }

    /* The kernel's state of one thread: where its fields live and its twiddles
     * (the interface drive() runs the round trips through). */
    struct Engine {
        using Math = Ssfm;
        C *home, *scratch;
        C *gf[3];
        StageTwiddles<M, C> tw;
        Staged *staged;
        Stager st;
        int t, rank;

        __device__ __forceinline__ void init(int)
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            C *const sm = reinterpret_cast<C *>(smem_raw);
            __shared__ Staged s_staged[F];
            home = GH ? nullptr : sm;
            scratch = GH ? sm : (INPLACE ? home : home + (size_t)F * M);
            staged = s_staged;
            t = threadIdx.x;
            rank = 0;
            if constexpr (CL > 1) rank = (int)cg::this_cluster().block_rank();
            C *twtab = sm + field_elems();
            fill_twiddle_table<M>(twtab, t);
            tw.init(t, twtab);
            __syncthreads();
        }

        /* every thread of the instance's CTAs */
        __device__ __forceinline__ void barrier() { bar(); }

        template <typename X>
        static __device__ __forceinline__ X *cta(X *p, int r)
        {
            return peer(p, r);
        }

        __device__ __forceinline__ void load(const Instance &I)
        {
            gf[0] = reinterpret_cast<C *>(I.Ap);
            gf[1] = reinterpret_cast<C *>(I.As);
            gf[2] = reinterpret_cast<C *>(I.Ai);
            if constexpr (!GH) {
#pragma unroll
                for (int f = 0; f < F; f++)
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        home[f * M + swz<C>(t + e * T)] = gf[f][(size_t)rank * M + t + e * T];
            }
            xsync();
        }

        __device__ __forceinline__ void store()
        {
            if constexpr (!GH) {
#pragma unroll
                for (int f = 0; f < F; f++)
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        gf[f][(size_t)rank * M + t + e * T] = home[f * M + swz<C>(t + e * T)];
            }
        }

        /* the field f of this CTA for the local transforms */
        __device__ __forceinline__ C *fld(int f) const
        {
            return GH ? gf[f] + (size_t)rank * M : home + (size_t)f * M;
        }

        /* Starts the loads of the next pass's coefficients; `now`: no
         * dispersion step comes before that pass. */
        __device__ __forceinline__ void stage(const Ops &op, const Tables &tab, bool now)
        {
            st.load(t - (T - 32), op, tab);
            if (now) {
                st.write(t - (T - 32), staged);
                __syncthreads();
            }
        }

        __device__ __forceinline__ void pass(unsigned in_y, unsigned out_y, Ops &op, const Instance &I,
                                             const Tables &tab, const RkConst<R> &rkc, int eom_idler, double (&th)[3],
                                             double &acc)
        {
            if (op.frame >= 0) frame_step(op, staged->c + 6, staged->u, th);
            cross(home, gf, in_y, out_y, op, I, tab, coef(staged, rkc), eom_idler, acc, t, rank);
            if (!op.power) xsync(); /* (power() synchronises) */
        }

        __device__ __forceinline__ void dispersion(const Tables &tab)
        {
            const C *__restrict__ disp = reinterpret_cast<const C *>(tab.disp);
            /* FP32, 2 equations: one copy of the code per field, so that one
             * field's last stores overlap the other's loads (333 instances of
             * 2^13: 9.3 ms against 10.1 with a loop), except in the kernels
             * of one CTA per SM (solo_f32_2eq.cu), which run side by side
             * with other grids' and share instruction caches (32 instances
             * of 2^12..2^15: 18.8 us per slice against 21.7 with a copy per
             * field).  Elsewhere one copy: the others gain nothing from more
             * (32 FP64 instances of 2^12..2^15: 31.5 us per slice against
             * 33.8). */
#pragma unroll COPIES
            for (int f = 0; f < F; f++) {
                spectral<0>(fld(f), scratch, disp + ((size_t)f * CL + rank) * M, nullptr, 0.0, 0.0, 0, tab.inv_n, tw,
                            t);
                /* copy 0 counts (the next field's exchanges make it visible); a
                 * test of f would split the loop */
                st.write(t - (T - 32), staged + f);
            }
            xsync();
        }

        __device__ __forceinline__ int failed() const { return 0; }
        __device__ __forceinline__ bool stopped() const { return false; }
        __device__ __forceinline__ int error() const { return 0; }
        __device__ __forceinline__ void drain() const {}

        __device__ __forceinline__ void gdd(const Tables &tab, const Instance &I)
        {
            /* (nothing is staged here: with CL = 1 no barrier lies between the
             * pass before this step, where every warp reads the coefficients,
             * and its start; the pass after it uses none) */
            const float *__restrict__ w = tab.w + (size_t)rank * M;
            spectral<1>(fld(1), scratch, nullptr, w, I.gdd, I.tod_s, I.use_tod_s, tab.inv_n, tw, t);
            if constexpr (F == 3)
                spectral<1>(fld(2), scratch, nullptr, w, I.gdd, I.tod_i, I.use_tod_i, tab.inv_n, tw, t);
            xsync();
        }

        /* Sum of the threads' acc over the cluster, the same on every CTA.
         * The order is fixed by the grid alone, not by the thread layout:
         * each (CTA rank, t) adds its points in order (acc), then 16
         * consecutive t by xor, then the groups of 16, then the ranks. */
        __device__ __forceinline__ double power(double acc)
        {
            __shared__ double red[32];
            __shared__ double red_cl;
            double v = acc;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((t & 15) == 0) red[t >> 4] = v;
            __syncthreads();
            double part = 0.0;
#pragma unroll
            for (int q = 0; q < T / 16; q++) part += red[q];
            __syncthreads();
            if constexpr (CL > 1) {
                if (t == 0) red_cl = part;
                csync();
                part = 0.0;
#pragma unroll
                for (int c = 0; c < CL; c++) part += *peer(&red_cl, c);
            }
            return part;
        }
    };
};

/*
 * The round trips of the instances of one launch.  Engine: the kernel's thread
 * layout (where the fields live, how a pass over them is spread over threads
 * and CTAs); Engine::Math: the arithmetic.  Control flow is uniform over the
 * threads of an instance.
 */
template <typename R, class Engine>
static __device__ __forceinline__ void drive(const LaunchArgs &a)
{
    using K = typename Engine::Math;
    using C = cpx<R>;
    using Ops = typename K::Ops;
    constexpr int N = K::N, NCO = K::NCO;
    constexpr unsigned ALL = K::ALL;
    __shared__ int next_inst;
    Engine E;
    E.init(a.hold);
    bool first = true;
    for (;;) {
        int idx;
        if (a.inst) {
            if (E.rank == 0 && threadIdx.x == 0) next_inst = atomicAdd(a.queue, 1);
            E.barrier();
            idx = *E.cta(&next_inst, 0);
            E.barrier();
            if (idx >= a.n_inst) break;
        } else {
            if (!first) break;
            idx = 0;
        }
        first = false;
        const bool leader = E.rank == 0 && threadIdx.x == 0;
        const Instance &I = a.inst ? a.inst[idx] : a.single;
        /* this instance's tables: its own where it has them, else the launch's */
        Tables tab = a.tab;
        int use_eom = a.use_eom;
        if (I.disp) {
            tab.disp = I.disp;
            tab.rk = I.rk;
            tab.w = I.w;
            tab.h6 = I.h6;
            tab.kp = I.kp;
            tab.ks = I.ks;
            tab.g_last = I.g_last;
            tab.eom = I.eom;
            use_eom = I.eom != nullptr;
        }
        RkConst<R> rkc;
        rkc.hp = (R)(0.5 * tab.kp);
        rkc.hs = (R)(0.5 * tab.ks);
        rkc.fp = (R)tab.kp;
        rkc.fs = (R)tab.ks;
        rkc.gp = (R)(tab.h6 * tab.kp);
        rkc.gs = (R)(tab.h6 * tab.ks);
        const C *__restrict__ rk = reinterpret_cast<const C *>(tab.rk);
        int rt_begin = I.rt_begin, rt_count = I.rt_count, patience = I.patience, calm = 0;
        double tol = I.tol, prev_ps = -1.0;
        if (I.st_flag) {
            /* batch instance: resume from its saved state, skip if done */
            if (*(volatile int *)I.st_flag != 0) continue;
            rt_begin = *(volatile int *)I.st_rt;
            rt_count = min(a.chunk, K::rt_limit(a, I) - rt_begin);
            prev_ps = rt_begin > 0 ? *(volatile double *)I.st_ps : -1.0;
            calm = *(volatile int *)I.st_calm;
            tol = a.tol;
            patience = a.patience;
        }
        /* no round trip left: without a round trip's barriers, all threads of
         * the instance must still have read its state before the leader
         * writes it below */
        if (rt_count < 1) E.barrier();
        E.load(I);

        double ps = prev_ps, acc = 0.0;
        int rts = 0, flag = 0;
        bool stop = false;
        for (int rt = rt_begin; rt < rt_begin + rt_count && !stop; rt++) {
            double th[3] = {tab.g_last, 0.0, 0.0};
            {
                Ops op{};
                op.inject = !a.pass_only;
                if (a.regime == 1) {
                    /* ReadPump offsets, functions.cuh:196-210 (Q6) */
                    const int nrt = I.n_rt_total;
                    op.poff = (rt == 0) ? 0 : ((rt > 0 && rt < nrt - 1) ? (long)rt * N : (long)N * nrt - 1 - N);
                }
                op.turn = rk + (size_t)a.n_z * NCO;
                op.rk1 = rk;
                op.frame = frame_index(rt, 0);
                E.stage(op, tab, true);
                E.pass(0u, ALL, op, I, tab, rkc, a.eom_idler, th, acc);
            }
            /* the pass after the dispersion step of slice s */
            auto between = [&](int s) {
                Ops op{};
                op.frame = -1;
                op.rk0 = rk + (size_t)s * NCO;
                if (s + 1 < a.n_z) {
                    op.turn = op.rk0;
                    op.rk1 = op.rk0 + NCO;
                    op.frame = frame_index(rt, s + 1);
                }
                return op;
            };
            for (int s = 0; s < a.n_z && !E.stopped(); s++) {
                E.stage(between(s), tab, false);
                E.dispersion(tab);
                if (s + 1 < a.n_z) {
                    Ops op = between(s);
                    E.pass(ALL, ALL, op, I, tab, rkc, a.eom_idler, th, acc);
                }
            }
            rts++;
            Ops end = between(a.n_z - 1);
            if (a.pass_only) {
                K::frame_back(end, th);
                E.pass(ALL, 0u, end, I, tab, rkc, a.eom_idler, th, acc);
                break;
            }
            unsigned in_y = ALL;
            end.eom = use_eom;
            if (I.gdd != 0.0) {
                /* GDD / TOD compensation of the resonant fields (cuOPO.cu:521-553):
                 * signal and idler go to the frequency domain, the pump stays in time */
                in_y = ALL & ~1u;
                E.pass(ALL, in_y, end, I, tab, rkc, a.eom_idler, th, acc);
                end = Ops{};
                end.frame = -1;
                E.gdd(tab, I);
            }
            const bool save = (rt >= I.save_first && rt < I.save_first + I.save_count);
            end.addphase = 1;
            end.ph_s = make_double2(I.phase_s[0], I.phase_s[1]);
            end.ph_i = make_double2(I.phase_i[0], I.phase_i[1]);
            end.save = save;
            end.slot = save ? (size_t)(rt - I.save_first) * N : 0;
            end.power = 1;
            acc = 0.0;
            K::frame_back(end, th);
            E.pass(in_y, 0u, end, I, tab, rkc, a.eom_idler, th, acc);
            ps = E.power(acc) * tab.inv_n;
            /* single launches record from rt_begin, batch instances by round trip */
            if (leader && I.ps_hist) I.ps_hist[I.st_flag ? rt : rt - rt_begin] = ps;
            if (!(ps == ps) || ps > 1.0e300) {
                if (leader && a.status) atomicCAS(a.status, 0, (int)ST_NONFINITE);
                flag = ST_NONFINITE;
                stop = true;
            }
            /* convergence: relative change of the signal power per rt below
             * tol for `patience` consecutive rts (from the second rt on) */
            if (tol > 0.0 && prev_ps > 0.0 && ps > 0.0 && fabs(ps - prev_ps) < tol * ps) {
                if (++calm >= (patience > 0 ? patience : 1) && flag == 0) {
                    flag = ST_CONVERGED;
                    stop = true;
                }
            } else {
                calm = 0;
            }
            prev_ps = ps;
            if (E.error()) {
                flag = ST_TIMEOUT;
                stop = true;
            }
        }
        E.store();
        if (threadIdx.x == 0 && E.failed() && a.status) atomicCAS(a.status, 0, (int)ST_TIMEOUT);
        if (leader) {
            if (I.rt_done) *I.rt_done = rts;
            if (I.ps_out) *I.ps_out = ps;
            if (I.flag_out) *I.flag_out = flag;
            if (I.st_flag) {
                *I.st_rt = rt_begin + rts;
                *I.st_ps = ps;
                *I.st_calm = calm;
                *I.st_flag = flag != 0 ? flag : (rt_begin + rts >= K::rt_limit(a, I) ? (int)ST_LIMIT : 0);
            }
        }
        E.barrier();
        if (E.failed() || E.error()) {
            /* this cluster's exchanges are out of step: instances that it has
             * not taken stay as they are, for another cluster or a later
             * launch.  Nothing may still be on its way to a CTA that exits. */
            E.drain();
            break;
        }
    }
}

template <typename R, int F, int M, int CL, int HM, int MINB, int COPIES = field_copies<R>(F)>
__global__ void __launch_bounds__(M / 16, MINB) ssfm_kernel(LaunchArgs a)
{
    drive<R, typename Ssfm<R, F, M, CL, HM, COPIES>::Engine>(a);
}

}  // namespace cuopo
