/*
 * wide.cuh -- the SSFM round trips of ONE instance spread over a cluster of P
 * CTAs: for launches of few instances, where ssfm_kernel leaves most of the
 * chip idle and each slice is a serial chain through one CTA (or a few).
 *
 * The arithmetic is that of Ssfm<R, F, M, CL>, operation for operation: the
 * same Stockham stages (radix R0, 16, 16 on M points, R0 = M/256), the same
 * radix-CL cross stage and the same element-wise passes, so the results are
 * equal bit for bit and either kernel may run an instance.  Only the
 * distribution differs.  The first forward stage (radix R0) and the last
 * inverse stage (radix 16) combine points n1 that agree mod T = M/16, and so
 * do the cross stage (all CL values of one n1) and the element-wise pass.
 * What lies between them are independent 256-point transforms, one per
 * (field, cross index k2, first-stage output r).  So
 *
 *   time side: CTA p owns the classes n1 mod T in [p Tc, (p+1) Tc),
 *     Tc = T/P: the last inverse stage, cross stage, RK4 steps, cross stage
 *     and first forward stage need no other CTA;
 *   frequency side: CTA p owns the 256-point transforms r in
 *     [p R0/P, (p+1) R0/P) of every k2: two forward stages, the dispersion
 *     factor and two inverse stages run in 16 lanes each, with warp
 *     synchronisation alone;
 *
 * and each slice has two exchanges over distributed shared memory.  An
 * exchange is pushed: every thread stores its outputs into the owner's
 * buffer with st.async, which counts the bytes on the owner's mbarrier, and
 * the owner waits for its own bytes only.  No cluster barrier is needed
 * between slices (an arrive.release / wait.acquire pair of 16 CTAs took
 * 1.1 us of a slice's 4.8 at 2^13 points): a buffer may be overwritten once
 * its owner's next contribution to the sender has arrived, because every
 * thread of the owner reads its part before it sends, and every thread sends
 * to every CTA.
 *
 * Every 16-point transform is one thread's, all fields at once, so a CTA has
 * F CL 16 R0/P transform threads; the element-wise pass uses all NTHR of the
 * CTA.  The chain per slice is what bounds it (six 16-point transforms, two
 * exchanges, two RK4 half steps), so whatever does not depend on the fields
 * is loaded ahead: the pass's coefficients by the last warp into shared
 * memory before the dispersion step (stage()), the dispersion rows and the
 * stage rotations before the wait or, where registers allow, once.
 *
 * The waits are bounded (1 s of %globaltimer): one that gives up marks the
 * CTA, all its later waits return at once, and the instance ends with
 * ST_TIMEOUT after the round trip, on every CTA of the cluster.
 */
#pragma once
#include "ssfm.cuh"

namespace cuopo {

/* Stores to the shared memory of a cluster's CTA (address from mapa). */
__device__ __forceinline__ unsigned smem_addr(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned map_cta(unsigned addr, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

/* Asynchronous stores that count their bytes on an mbarrier of the same CTA. */
__device__ __forceinline__ void st_async(unsigned addr, unsigned mbar, float2 v)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void st_async(unsigned addr, unsigned mbar, double2 v)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(v.x), "d"(v.y), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned mbar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
}

template <typename R, int F, int M, int CL, int P, int NTHR, int MINB>
struct Wide {
    using Math = Ssfm<R, F, M, CL, 0>;
    using C = cpx<R>;
    using SP = StagePlan<M>;
    using Ops = typename Math::Ops;
    static constexpr int T = SP::T, N = M * CL, R0 = SP::R0;
    static constexpr int B = 16 / R0;        /* first-stage butterflies per 16 points */
    static constexpr int Tc = T / P;         /* classes of a CTA */
    static constexpr int RP = R0 / P;        /* first-stage outputs r of a CTA */
    static constexpr int U = CL * RP;        /* 256-point transforms per field of a CTA */
    static constexpr int NP = 16 * Tc;       /* positions n1 of a CTA */
    static constexpr int NT = F * CL * Tc;   /* transform threads (= F U 16) */
    static constexpr unsigned ALL = Math::ALL;
    /* cross stages of 16 values of every field do not fit a thread's
     * registers beside the RK4 step: one field at a time there */
    static constexpr bool SPLIT = CL == 16;
    static_assert(SP::P == 3, "radix R0, 16, 16 only");
    static_assert(R0 % P == 0 && P <= 16 && NTHR % 32 == 0 && NT % 16 == 0, "cluster size divides the first radix");

    /* stage rotations and dispersion rows kept in registers */
    static constexpr bool HOLD_TW = sizeof(R) == 4 && NT <= NTHR && NTHR * MINB <= 256;
    static constexpr bool EARLY_ROWS = NTHR * MINB <= 256;

    static constexpr size_t buf_elems() { return (size_t)F * CL * NP; }
    static constexpr size_t smem_bytes() { return sizeof(C) * 2 * buf_elems(); }

    /* One 16-point transform.  Time side: field, cross index, class;
     * frequency side: field, transform (uk2, r), lane.  The field is the same on
     * both sides (task / (CL Tc) == task / (16 U)). */
    struct Role {
        int f, k2, t2l, uu, uk2, r, lane;
        __device__ __forceinline__ Role(int task, int rank)
        {
            f = task / (Tc * CL);
            k2 = (task / Tc) % CL;
            t2l = task % Tc;
            uu = task >> 4;
            uk2 = (uu % U) / RP;
            r = rank * RP + uu % RP;
            lane = task & 15;
        }
        /* rotations of the time side's inverse stage and of the frequency side's twiddled stages */
        __device__ __forceinline__ StageRot<C> rot_t(int rank) const { return load_rot(tw_row<C>(rank * Tc + t2l, T)); }
        __device__ __forceinline__ StageRot<C> rot_1() const { return load_rot(tw_row<C>(r, R0)); }
        __device__ __forceinline__ StageRot<C> rot_2() const { return load_rot(tw_row<C>(r + R0 * lane, T)); }
        __device__ __forceinline__ StageRot<C> rot_3() const { return load_rot(tw_row<C>(lane % R0, R0)); }
    };

    struct Engine {
        using Math = Wide::Math;
        C *tb;      /* [F][CL][16][Tc]: time side, point t2 + T e + M c at [f][c][e][t2 - rank Tc] */
        C *fb;      /* [F][U][256]: frequency side, entry j of transform (k2, r) */
        C *gf[3];
        unsigned long long *mbar;  /* [3 b + f]: field f of buffer b (0: tb, 1: fb) */
        int *dead;                 /* [0]: a wait of this CTA gave up; [1 + c]: CTA c's, after power() */
        typename Math::Staged *staged;
        typename Math::Stager st;
        unsigned parity;           /* bit 3 b + f: parity of that mbarrier's next phase */
        int tid, rank;
        StageRot<C> w_t, w_1, w_2, w_3; /* HOLD_TW: this thread's rotations */

        __device__ __forceinline__ void init()
        {
            extern __shared__ __align__(16) unsigned char smem_raw[];
            __shared__ unsigned long long s_mbar[6];
            __shared__ int s_dead[1 + P];
            __shared__ typename Math::Staged s_staged;
            tb = reinterpret_cast<C *>(smem_raw);
            fb = tb + buf_elems();
            mbar = s_mbar;
            dead = s_dead;
            staged = &s_staged;
            parity = 0;
            tid = threadIdx.x;
            rank = 0;
            if constexpr (P > 1) rank = (int)cg::this_cluster().block_rank();
            if (tid <= P) s_dead[tid] = 0;
            if constexpr (P > 1) {
                if (tid < 6)
                    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_mbar[tid])) : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            if constexpr (HOLD_TW) {
                const Role o(tid, rank);
                w_t = o.rot_t(rank);
                w_1 = o.rot_1();
                w_2 = o.rot_2();
                w_3 = o.rot_3();
            }
            /* every CTA of the cluster runs, its barriers initialised, before the first store to it */
            barrier();
        }

        __device__ __forceinline__ void barrier()
        {
            if constexpr (P > 1) Math::csync();
            else __syncthreads();
        }

        template <typename X>
        static __device__ __forceinline__ X *cta(X *p, int c)
        {
            if constexpr (P == 1) return p;
            else return cg::this_cluster().map_shared_rank(p, c);
        }

        /* buf[i] of CTA c's shared memory = v, counted on its mbar[m] */
        __device__ __forceinline__ void put(C *buf, int m, int c, int i, C v)
        {
            if constexpr (P == 1) buf[i] = v;
            else
                st_async(map_cta(smem_addr(buf), c) + (unsigned)(i * (int)sizeof(C)), map_cta(smem_addr(mbar + m), c),
                         v);
        }

        /* Announces this CTA's bytes of the exchange into buffer b, per field of mask. */
        __device__ __forceinline__ void expect(int b, unsigned mask)
        {
            if constexpr (P > 1) {
                if (tid < F && ((mask >> tid) & 1u))
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                     smem_addr(mbar + 3 * b + tid)),
                                 "r"((unsigned)(CL * NP * (int)sizeof(C)))
                                 : "memory");
            }
        }

        /* Waits for field f of the exchange into buffer b (the threads that
         * read it; then flip() by all, for the fields of the exchange). */
        __device__ __forceinline__ void wait(int b, int f)
        {
            if constexpr (P > 1) {
                const unsigned m = smem_addr(mbar + 3 * b + f), par = (parity >> (3 * b + f)) & 1u;
                if (mbar_test(m, par)) return;
                unsigned long long t0, t1;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
                while (!mbar_test(m, par)) {
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
                    if (*(volatile int *)dead || t1 - t0 > 1000000000ull) {
                        *(volatile int *)dead = 1;
                        return;
                    }
                }
            }
        }
        __device__ __forceinline__ void flip(int b, unsigned mask) { parity ^= mask << (3 * b); }

        /* a wait of this CTA gave up */
        __device__ __forceinline__ int failed() const { return P > 1 ? *(volatile int *)dead : 0; }

        /* a wait of any CTA gave up (the same on every CTA, after power()) */
        __device__ __forceinline__ int error() const
        {
            int e = 0;
            if constexpr (P > 1) {
#pragma unroll
                for (int c = 0; c < P; c++) e |= dead[1 + c];
            }
            return e;
        }

        /* Starts the loads of the next pass's coefficients (pass() writes them
         * to shared memory before its first barrier). */
        __device__ __forceinline__ void stage(const Ops &op, const Tables &tab, bool)
        {
            st.load(tid - (NTHR - 32), op, tab);
        }

        /* index into the global fields of entry i (position and cross index) of the time side */
        __device__ __forceinline__ int point(int pos, int c) const
        {
            return rank * Tc + pos % Tc + T * (pos / Tc) + M * c;
        }

        __device__ __forceinline__ void load(const Instance &I)
        {
            gf[0] = reinterpret_cast<C *>(I.Ap);
            gf[1] = reinterpret_cast<C *>(I.As);
            gf[2] = reinterpret_cast<C *>(I.Ai);
#pragma unroll
            for (int q = 0; q < F; q++)
                for (int i = tid; i < CL * NP; i += NTHR) tb[q * CL * NP + i] = gf[q][point(i % NP, i / NP)];
            __syncthreads();
        }

        __device__ __forceinline__ void store()
        {
#pragma unroll
            for (int q = 0; q < F; q++)
                for (int i = tid; i < CL * NP; i += NTHR) gf[q][point(i % NP, i / NP)] = tb[q * CL * NP + i];
        }

        /* A pass over the time side: the fields of in_y come from the
         * exchange (last inverse stage and inverse cross stage first), those
         * of out_y go on (cross stage, first forward stage, exchange). */
        __device__ __forceinline__ void pass(unsigned in_y, unsigned out_y, Ops &op, const Instance &I,
                                             const Tables &tab, const RkConst<R> &rkc, int eom_idler, double (&th)[3],
                                             double &acc)
        {
            const C *__restrict__ twN = reinterpret_cast<const C *>(tab.twN);
            st.write(tid - (NTHR - 32), staged);
            if (in_y) {
#pragma unroll 1
                for (int task = tid; task < NT; task += NTHR) {
                    const Role o(task, rank);
                    if (!((in_y >> o.f) & 1u)) continue;
                    C *const own = tb + (o.f * CL + o.k2) * NP + o.t2l;
                    const int t2 = rank * Tc + o.t2l;
                    StageRot<C> w;
                    if constexpr (HOLD_TW) w = w_t;
                    else w = o.rot_t(rank);
                    C v[16];
                    wait(0, o.f);
#pragma unroll
                    for (int e = 0; e < 16; e++) v[e] = own[e * Tc];
                    dft16<-1, true>(v, w, 2 * t2 >= T);
#pragma unroll
                    for (int e = 0; e < 16; e++) own[e * Tc] = v[e];
                }
                flip(0, in_y);
            }
            __syncthreads();
            const typename Math::Coef co = Math::coef(staged, rkc);
            if (op.frame >= 0) Math::frame_step(op, staged->c + 6, staged->u, th);
            if (out_y) expect(1, out_y);
            if constexpr (SPLIT) {
                cross_field<-1>(in_y, twN);
                __syncthreads();
#pragma unroll 1
                for (int i = tid; i < CL * NP; i += NTHR) {
                    C A[3];
#pragma unroll
                    for (int q = 0; q < F; q++) A[q] = tb[q * CL * NP + i];
                    Math::pointwise(A, point(i % NP, i / NP), op, co, I, tab, eom_idler, acc);
#pragma unroll
                    for (int q = 0; q < F; q++) tb[q * CL * NP + i] = A[q];
                }
                __syncthreads();
                cross_field<+1>(out_y, twN);
            } else {
#pragma unroll 1
                for (int pos = tid; pos < NP; pos += NTHR) {
                    C v[3][CL];
#pragma unroll
                    for (int q = 0; q < F; q++)
#pragma unroll
                        for (int c = 0; c < CL; c++) v[q][c] = tb[(q * CL + c) * NP + pos];
                    const int n1 = point(pos, 0);
                    if constexpr (CL > 1) {
#pragma unroll
                        for (int q = 0; q < F; q++)
                            if ((in_y >> q) & 1u) Math::cross_inv(v[q], n1, twN);
                    }
#pragma unroll
                    for (int c = 0; c < CL; c++) {
                        C A[3];
#pragma unroll
                        for (int q = 0; q < F; q++) A[q] = v[q][c];
                        Math::pointwise(A, n1 + M * c, op, co, I, tab, eom_idler, acc);
#pragma unroll
                        for (int q = 0; q < F; q++) v[q][c] = A[q];
                    }
                    if constexpr (CL > 1) {
#pragma unroll
                        for (int q = 0; q < F; q++)
                            if ((out_y >> q) & 1u) Math::cross_fwd(v[q], n1, twN);
                    }
#pragma unroll
                    for (int q = 0; q < F; q++)
#pragma unroll
                        for (int c = 0; c < CL; c++) tb[(q * CL + c) * NP + pos] = v[q][c];
                }
            }
            __syncthreads();
            if (!out_y) return;
#pragma unroll 1
            for (int task = tid; task < NT; task += NTHR) {
                const Role o(task, rank);
                if (!((out_y >> o.f) & 1u)) continue;
                const C *const own = tb + (o.f * CL + o.k2) * NP + o.t2l;
                C v[16];
#pragma unroll
                for (int e = 0; e < 16; e++) v[e] = own[e * Tc];
                first_stage<+1>(v);
#pragma unroll
                for (int q = 0; q < R0; q++) /* output q of butterfly i: entry t2 + T i of transform (k2, q) */
#pragma unroll
                    for (int i = 0; i < B; i++)
                        put(fb, 3 + o.f, q / RP, (o.f * U + o.k2 * RP + q % RP) * 256 + rank * Tc + o.t2l + T * i,
                            v[i + q * B]);
            }
            if constexpr (P == 1) __syncthreads();
        }

        /* The radix-CL stage of one field at one position per thread (SPLIT). */
        template <int S>
        __device__ __forceinline__ void cross_field(unsigned mask, const C *__restrict__ twN)
        {
#pragma unroll 1
            for (int i = tid; i < F * NP; i += NTHR) {
                const int q = i / NP, pos = i % NP;
                if (!((mask >> q) & 1u)) continue;
                C v[CL];
#pragma unroll
                for (int c = 0; c < CL; c++) v[c] = tb[(q * CL + c) * NP + pos];
                if constexpr (S < 0) Math::cross_inv(v, point(pos, 0), twN);
                else Math::cross_fwd(v, point(pos, 0), twN);
#pragma unroll
                for (int c = 0; c < CL; c++) tb[(q * CL + c) * NP + pos] = v[c];
            }
        }

        template <int S>
        static __device__ __forceinline__ void first_stage(C (&v)[16])
        {
            stage_compute<S, M, 0>(v, StageTwiddles<M, C>{});
        }

        /* The frequency side of the fields of mask: two forward stages, the
         * factor, two inverse stages, exchange.  MODE as Ssfm::spectral. */
        template <int MODE>
        __device__ __forceinline__ void spectral(unsigned mask, const Tables &tab, const Instance *I)
        {
            expect(0, mask);
#pragma unroll 1
            for (int task = tid; task < NT; task += NTHR) {
                const Role o(task, rank);
                if (!((mask >> o.f) & 1u)) continue;
                const int r = o.r, lane = o.lane, t2p = r + R0 * lane;
                const unsigned half = 0xFFFFu << (tid & 16); /* the transform's 16 lanes */
                C *const u = fb + o.uu * 256;
                /* row entries of frequencies t2p + T e, [k2][r][e][lane] */
                const int row = ((o.uk2 * R0 + r) * 16) * 16 + lane;
                const C *__restrict__ disp = reinterpret_cast<const C *>(tab.disp) + (size_t)o.f * N + row;
                C v[16], d[EARLY_ROWS ? 16 : 1];
                if constexpr (MODE == 0 && EARLY_ROWS) {
#pragma unroll
                    for (int e = 0; e < 16; e++) d[e] = ld_now(disp + 16 * e);
                }
                wait(1, o.f);
                /* stage 1 (length R0): butterfly `lane`, k = r */
#pragma unroll
                for (int e = 0; e < 16; e++) v[e] = u[lane + 16 * e];
                if constexpr (HOLD_TW) dft16<+1, true>(v, w_1, 2 * r >= R0);
                else dft16<+1, true>(v, o.rot_1(), 2 * r >= R0);
                __syncwarp(half);
#pragma unroll
                for (int q = 0; q < 16; q++) u[16 * q + (lane ^ q)] = v[q];
                __syncwarp(half);
                /* stage 2 (length T): butterfly t2p = r + R0 lane; leaves frequencies t2p + T e */
#pragma unroll
                for (int e = 0; e < 16; e++) v[e] = u[16 * lane + (e ^ lane)];
                if constexpr (HOLD_TW) dft16<+1, true>(v, w_2, 2 * t2p >= T);
                else dft16<+1, true>(v, o.rot_2(), 2 * t2p >= T);
                const R s_n = (R)tab.inv_n;
                if constexpr (MODE == 0) {
#pragma unroll
                    for (int e = 0; e < 16; e++)
                        v[e] = caddmul(cscale(v[e], s_n), EARLY_ROWS ? d[e % (EARLY_ROWS ? 16 : 1)]
                                                                     : __ldg(disp + 16 * e));
                } else {
                    Math::gdd_factor(v, tab.w + row, 16, I->gdd, o.f == 1 ? I->tod_s : I->tod_i,
                                     o.f == 1 ? I->use_tod_s : I->use_tod_i, s_n);
                }
                /* inverse stage 0 (radix R0) on the same registers */
                first_stage<-1>(v);
                __syncwarp(half);
                /* to butterfly s = q R0 + r0, element e1: (position R0 j + r0, j = t2p + T i = 16 e1 + r + R0 q) */
#pragma unroll
                for (int r0 = 0; r0 < R0; r0++)
#pragma unroll
                    for (int i = 0; i < B; i++) {
                        const int s = (lane % B) * R0 + r0, e1 = lane / B + R0 * i;
                        u[16 * e1 + (s ^ e1)] = v[i + r0 * B];
                    }
                __syncwarp(half);
                const int k = lane % R0, q = r + R0 * (lane / R0);
#pragma unroll
                for (int e = 0; e < 16; e++) v[e] = u[16 * e + (lane ^ e)];
                if constexpr (HOLD_TW) dft16<-1, true>(v, w_3, 2 * k >= R0);
                else dft16<-1, true>(v, o.rot_3(), 2 * k >= R0);
                /* output m: element q of class k + R0 m */
#pragma unroll
                for (int m = 0; m < 16; m++) {
                    const int c = k + R0 * m;
                    put(tb, o.f, c / Tc, (o.f * CL + o.uk2) * NP + q * Tc + c % Tc, v[m]);
                }
            }
            flip(1, mask);
            if constexpr (P == 1) __syncthreads();
        }

        __device__ __forceinline__ void dispersion(const Tables &tab) { spectral<0>(ALL, tab, nullptr); }

        __device__ __forceinline__ void gdd(const Tables &tab, const Instance &I)
        {
            spectral<1>(ALL & ~1u, tab, &I);
        }

        /* Sum of |As|^2 in Ssfm's order: partial sums per (CTA rank of that
         * layout, t), 16 consecutive t by xor, the groups, the ranks.  pass()
         * has left the signal on the time side. */
        __device__ __forceinline__ double power(double)
        {
            constexpr int J = 16 / CL, G = T / 16;
            __shared__ double red[CL * G];
            static_assert(CL * Tc <= NTHR, "one partial sum per thread");
            if (tid < CL * Tc) {
                const int rk = tid / Tc, t2l = tid % Tc; /* that layout's rank, class */
                double v = 0.0;
#pragma unroll
                for (int j = 0; j < J; j++)
#pragma unroll
                    for (int c = 0; c < CL; c++) v += cabs2d(tb[(CL + c) * NP + (rk * J + j) * Tc + t2l]);
                const unsigned half = 0xFFFFu << (tid & 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(half, v, o);
                const int g = rank * (Tc / 16) + t2l / 16;
                if ((tid & 15) < P) *cta(&red[rk * G + g], tid & 15) = v;
            }
            if constexpr (P > 1) {
                if (tid < P) *cta(&dead[1 + rank], tid) = *(volatile int *)dead;
            }
            barrier();
            double part = 0.0;
#pragma unroll
            for (int c = 0; c < CL; c++) {
                double s = 0.0;
#pragma unroll
                for (int g = 0; g < G; g++) s += red[c * G + g];
                part += s;
            }
            return part;
        }
    };
};

template <typename R, int F, int M, int CL, int P, int NTHR, int MINB>
__global__ void __launch_bounds__(NTHR, MINB) wide_kernel(LaunchArgs a)
{
    drive<R, typename Wide<R, F, M, CL, P, NTHR, MINB>::Engine>(a);
}

}  // namespace cuopo
