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
 * A CTA has F CL 16 R0/P 16-point transforms of every stage, all fields at
 * once; Q threads (1 or 4) do one.  With Q = 4 thread q holds the elements
 * e = q mod 4: the inner 4-point transforms over a are its own, and their
 * outputs change places within the quad through shared memory (the outer
 * ones, over b, then leave it the outputs q mod 4).  That is a quarter of the
 * instructions in each link of the chain: where a CTA has only a warp or two of
 * transforms (2^13 points or less on 16 CTAs) the others would idle.  The
 * element-wise pass uses all NTHR threads of the CTA.  The chain per slice is what bounds it (six 16-point transforms, two
 * exchanges, two RK4 half steps), so whatever does not depend on the fields
 * is loaded ahead: the pass's coefficients by the last warp into shared
 * memory before the dispersion step (stage()), the dispersion rows and the
 * stage rotations before the wait or, where registers allow, once.
 *
 * The waits are bounded (1 s of %globaltimer).  One that gives up marks the
 * CTA, whose other waits then give up at once.  The barrier's phase is
 * incomplete with no arrival pending, and another arrival is undefined, so
 * from the next pass on the CTA announces nothing any more and its slices end
 * (stopped(): read once per pass and used at the loop's own test; tests beside
 * the sends cost 2..4 % of a slice).  Its partners miss its bytes and give up
 * in their turn, so none gets more than two exchanges ahead of another.  The
 * instance ends with ST_TIMEOUT after the round trip, on every CTA of the
 * cluster, and the cluster takes no further one: it lets the stores under way
 * land (drain()) and exits.
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

/* dft16 by a quad: v[a] = element q + 4a in, output q + 4a out.  scr: the
 * warp's 128 entries of shared memory; tw: quarter turns and rotation of
 * W16^{b q}, b = 1..3 (QuadTw). */
template <typename C>
struct QuadTw {
    C rot[3];
    int m[3];
    __device__ __forceinline__ void init(int q)
    {
        using R = typename real_of<C>::type;
#pragma unroll
        for (int b = 1; b < 4; b++) {
            /* as tw16: n = b q eighths of pi, nearest quarter turn, rest r pi/8 with r = -1..2 */
            const int n = b * q, k = (n + 1) / 4, r = n - 4 * k;
            const double t = r == 0 ? 0.0 : r == 2 ? 0.41421356237309504880 : 0.19891236737965800691;
            const double sn = r == 0 ? 0.0 : r == 2 ? 0.70710678118654752440 : 0.38268343236508977173;
            rot[b - 1] = mk<C>((R)(r < 0 ? -t : t), (R)(r < 0 ? -sn : sn));
            m[b - 1] = k;
        }
    }
};

template <int S, bool TW, typename C>
__device__ __forceinline__ void dft16_quad(C (&v)[4], const StageRot<C> &w, bool hi, const QuadTw<C> &tw, C *scr)
{
    using R = typename real_of<C>::type;
    const R sg = (R)S;
    if constexpr (TW) {
        v[1] = shear_rot(v[1], sg * w.a[0].x, sg * w.a[0].y);
        v[2] = shear_rot(iq<S>(v[2]), sg * w.a[1].x, sg * w.a[1].y);
        v[3] = shear_rot(iq12<S>(v[3], hi), sg * w.a[2].x, sg * w.a[2].y);
    }
    dft4<S>(v[0], v[1], v[2], v[3]);
    /* 4 x 4 transpose: (q1, b) at 16 quad + ((4 q1 + b) ^ 4 (quad mod 4)) */
    const int l = threadIdx.x & 31, q = l & 3, base = (l >> 2) * 16, x = (l >> 2) & 3;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; j++) scr[base + 4 * (j ^ x) + q] = v[j];
    __syncwarp();
#pragma unroll
    for (int b = 0; b < 4; b++) v[b] = scr[base + 4 * (q ^ x) + b];
#pragma unroll
    for (int b = 1; b < 4; b++) {
        v[b] = shear_rot(iq_rt(v[b], (S * tw.m[b - 1]) & 3), sg * tw.rot[b - 1].x, sg * tw.rot[b - 1].y);
        if constexpr (TW) v[b] = shear_rot(v[b], sg * w.b[b - 1].x, sg * w.b[b - 1].y);
    }
    dft4<S>(v[0], v[1], v[2], v[3]);
}

template <typename R, int F, int M, int CL, int P, int NTHR, int MINB, int Q>
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
    static_assert(Q == 1 || (Q == 4 && 4 * NT <= NTHR && F * U <= 15), "quads: one transform each, a named barrier per 256 points");
    static constexpr int NV = 16 / Q;        /* elements of a thread */

    /* stage rotations and dispersion rows kept in registers */
    static constexpr bool HOLD_TW = sizeof(R) == 4 && Q * NT <= NTHR && (NTHR * MINB <= 256 || Q == 4);
    static constexpr bool EARLY_ROWS = NTHR * MINB <= 256 || Q == 4;

    static constexpr size_t buf_elems() { return (size_t)F * CL * NP; }
    static constexpr size_t smem_bytes() { return sizeof(C) * (2 * buf_elems() + (Q == 4 ? 4 * NTHR : 0)); }

    /* Places in the two buffers: quads read 8 neighbours of 4 elements e at a
     * time, so every other element is shifted by half of 16 entries (distinct
     * banks); in the exchange inside a 256-point transform, row and column of
     * a 16 x 16 matrix. */
    static __device__ __forceinline__ int tb_at(int e, int t2l) { return e * Tc + (Q == 4 ? t2l ^ (8 * (e & 1)) : t2l); }
    static __device__ __forceinline__ int fb_at(int j) { return Q == 4 ? j ^ ((j >> 1) & 8) : j; }
    static __device__ __forceinline__ int xc_at(int row, int col)
    {
        return 16 * row + (col ^ row ^ (Q == 4 ? 8 * (row & 1) : 0));
    }

    /* A 16-point transform, elements and outputs q + Q a of thread q. */
    template <int S, bool TW>
    static __device__ __forceinline__ void dft_q(C (&v)[NV], const StageRot<C> &w, bool hi, const QuadTw<C> &qt, C *scr)
    {
        if constexpr (Q == 1) dft16<S, TW>(v, w, hi);
        else dft16_quad<S, TW>(v, w, hi, qt, scr);
    }

    /* First forward (S = +1) or inverse stage, radix R0: butterflies i < B over
     * the elements i + B r.  Output j of thread q is output out_r(j, q) of
     * butterfly out_i(j, q). */
    template <int S>
    static __device__ __forceinline__ void first_stage(C (&v)[NV], const QuadTw<C> &qt, C *scr)
    {
        if constexpr (Q == 1) {
            stage_compute<S, M, 0>(v, StageTwiddles<M, C>{});
        } else if constexpr (R0 == 16) {
            dft16_quad<S, false>(v, StageRot<C>{}, false, qt, scr);
        } else if constexpr (R0 == 8) {
            /* dft8: b = q / 2, over a in the thread, then with the thread of the other b */
            dft4<S>(v[0], v[1], v[2], v[3]);
            const bool odd = (threadIdx.x & 2) != 0;
            C w[4] = {v[0], tw16<S, 2>(v[1]), tw16<S, 4>(v[2]), tw16<S, 6>(v[3])};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const C mine = odd ? w[k] : v[k];
                const C other = mk<C>(__shfl_xor_sync(0xffffffffu, mine.x, 2), __shfl_xor_sync(0xffffffffu, mine.y, 2));
                v[k] = odd ? csub(other, mine) : cadd(mine, other);
            }
        } else if constexpr (R0 == 4) {
            dft4<S>(v[0], v[1], v[2], v[3]);
        } else {
            dft2<S>(v[0], v[2]);
            dft2<S>(v[1], v[3]);
        }
    }
    static __device__ __forceinline__ int out_i(int j, int q)
    {
        if (Q == 1) return j % B;
        return R0 == 16 ? 0 : R0 == 8 ? (q & 1) : R0 == 4 ? q : q + 4 * (j & 1);
    }
    static __device__ __forceinline__ int out_r(int j, int q)
    {
        if (Q == 1) return j / B;
        return R0 == 16 ? q + 4 * j : R0 == 8 ? 4 * (q >> 1) + j : R0 == 4 ? j : j >> 1;
    }

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
        int gone;                  /* a wait of the CTA had given up by the latest pass (the same in every thread) */
        int tid, rank;
        int q;                     /* thread of the transform */
        QuadTw<C> qt;              /* Q == 4 */
        C *scr;
        StageRot<C> w_t, w_1, w_2, w_3; /* HOLD_TW: this thread's rotations */

        __device__ __forceinline__ void init(int hold)
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
            gone = 0;
            tid = threadIdx.x;
            rank = 0;
            if constexpr (P > 1) rank = (int)cg::this_cluster().block_rank();
            if (tid <= P) s_dead[tid] = 0;
            if constexpr (P > 1) {
                if (tid < 6)
                    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&s_mbar[tid])),
                                 "r"(hold && rank == 0 ? 0xFFFFF : 1) /* one arrival per exchange; held: never enough */
                                 : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            q = tid % Q;
            scr = fb + buf_elems() + (tid >> 5) * 128;
            if constexpr (Q == 4) qt.init(q);
            if constexpr (HOLD_TW) {
                const Role o(tid / Q, rank);
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

        /* Announces this CTA's bytes of the exchange into buffer b, per field of
         * mask; go: every wait before has succeeded (the barriers' phases are complete). */
        __device__ __forceinline__ void expect(int b, unsigned mask, bool go)
        {
            if constexpr (P > 1) {
                if (tid < F && ((mask >> tid) & 1u) && go)
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

        /* no further slices (the same in every thread of the CTA) */
        __device__ __forceinline__ bool stopped() const { return P > 1 && gone; }

        /* a wait of this CTA gave up */
        __device__ __forceinline__ int failed() const { return P > 1 ? *(volatile int *)dead : 0; }

        /* 2 ms for the stores under way to land in this CTA. */
        __device__ __forceinline__ void drain() const
        {
            unsigned long long t0, t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
            do asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            while (t1 - t0 < 2000000ull);
        }

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

        /* the threads of one 256-point transform */
        __device__ __forceinline__ void sync_unit(int uu)
        {
            if constexpr (Q == 1) __syncwarp(0xFFFFu << (tid & 16));
            else asm volatile("bar.sync %0, 64;" ::"r"(1 + uu) : "memory");
        }

        /* index into the global fields of entry pos (cross index c) of the time side */
        __device__ __forceinline__ int point(int pos, int c) const
        {
            const int e = pos / Tc;
            return rank * Tc + tb_at(e, pos % Tc) % Tc + T * e + M * c;
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
                for (int task = tid / Q; task < NT; task += NTHR / Q) {
                    const Role o(task, rank);
                    if (!((in_y >> o.f) & 1u)) continue;
                    C *const own = tb + (o.f * CL + o.k2) * NP;
                    const int t2 = rank * Tc + o.t2l;
                    StageRot<C> w;
                    if constexpr (HOLD_TW) w = w_t;
                    else w = o.rot_t(rank);
                    C v[NV];
                    wait(0, o.f);
#pragma unroll
                    for (int a = 0; a < NV; a++) v[a] = own[tb_at(q + Q * a, o.t2l)];
                    dft_q<-1, true>(v, w, 2 * t2 >= T, qt, scr);
#pragma unroll
                    for (int a = 0; a < NV; a++) own[tb_at(q + Q * a, o.t2l)] = v[a];
                }
                flip(0, in_y);
            }
            __syncthreads();
            gone = failed(); /* (no wait comes before the next barrier) */
            const typename Math::Coef co = Math::coef(staged, rkc);
            if (op.frame >= 0) Math::frame_step(op, staged->c + 6, staged->u, th);
            if (out_y) expect(1, out_y, !gone);
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
            for (int task = tid / Q; task < NT; task += NTHR / Q) {
                const Role o(task, rank);
                if (!((out_y >> o.f) & 1u)) continue;
                const C *const own = tb + (o.f * CL + o.k2) * NP;
                C v[NV];
#pragma unroll
                for (int a = 0; a < NV; a++) v[a] = own[tb_at(q + Q * a, o.t2l)];
                first_stage<+1>(v, qt, scr);
#pragma unroll
                for (int j = 0; j < NV; j++) { /* output k of butterfly i: entry t2 + T i of transform (k2, k) */
                    const int i = out_i(j, q), k = out_r(j, q);
                    put(fb, 3 + o.f, k / RP,
                        (o.f * U + o.k2 * RP + k % RP) * 256 + fb_at(rank * Tc + o.t2l + T * i), v[j]);
                }
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

        /* The frequency side of the fields of mask: two forward stages, the
         * factor, two inverse stages, exchange.  MODE as Ssfm::spectral. */
        template <int MODE>
        __device__ __forceinline__ void spectral(unsigned mask, const Tables &tab, const Instance *I)
        {
            if (MODE == 1 && gone) return;
            expect(0, mask, true); /* (not reached once gone: stopped() ends the slices) */
#pragma unroll 1
            for (int task = tid / Q; task < NT; task += NTHR / Q) {
                const Role o(task, rank);
                if (!((mask >> o.f) & 1u)) continue;
                const int r = o.r, lane = o.lane, t2p = r + R0 * lane;
                C *const u = fb + o.uu * 256;
                /* row entries of frequencies t2p + T e, [k2][r][e][lane] */
                const int row = ((o.uk2 * R0 + r) * 16 + q) * 16 + lane;
                const C *__restrict__ disp = reinterpret_cast<const C *>(tab.disp) + (size_t)o.f * N + row;
                C v[NV], d[EARLY_ROWS ? NV : 1];
                if constexpr (MODE == 0 && EARLY_ROWS) {
#pragma unroll
                    for (int a = 0; a < NV; a++) d[a] = ld_now(disp + 16 * Q * a);
                }
                wait(1, o.f);
                /* stage 1 (length R0): butterfly `lane`, k = r */
#pragma unroll
                for (int a = 0; a < NV; a++) v[a] = u[fb_at(lane + 16 * (q + Q * a))];
                if constexpr (HOLD_TW) dft_q<+1, true>(v, w_1, 2 * r >= R0, qt, scr);
                else dft_q<+1, true>(v, o.rot_1(), 2 * r >= R0, qt, scr);
                sync_unit(o.uu);
#pragma unroll
                for (int a = 0; a < NV; a++) u[xc_at(q + Q * a, lane)] = v[a];
                sync_unit(o.uu);
                /* stage 2 (length T): butterfly t2p = r + R0 lane; leaves frequencies t2p + T e */
#pragma unroll
                for (int a = 0; a < NV; a++) v[a] = u[xc_at(lane, q + Q * a)];
                if constexpr (HOLD_TW) dft_q<+1, true>(v, w_2, 2 * t2p >= T, qt, scr);
                else dft_q<+1, true>(v, o.rot_2(), 2 * t2p >= T, qt, scr);
                const R s_n = (R)tab.inv_n;
                if constexpr (MODE == 0) {
#pragma unroll
                    for (int a = 0; a < NV; a++)
                        v[a] = caddmul(cscale(v[a], s_n), EARLY_ROWS ? d[a % (EARLY_ROWS ? NV : 1)]
                                                                     : __ldg(disp + 16 * Q * a));
                } else {
                    Math::gdd_factor(v, tab.w + row, 16 * Q, I->gdd, o.f == 1 ? I->tod_s : I->tod_i,
                                     o.f == 1 ? I->use_tod_s : I->use_tod_i, s_n);
                }
                /* inverse stage 0 (radix R0) on the same registers */
                first_stage<-1>(v, qt, scr);
                sync_unit(o.uu);
                /* to butterfly s = q R0 + r0, element e1: (position R0 j + r0, j = t2p + T i = 16 e1 + r + R0 q) */
#pragma unroll
                for (int j = 0; j < NV; j++)
                    u[xc_at(lane / B + R0 * out_i(j, q), (lane % B) * R0 + out_r(j, q))] = v[j];
                sync_unit(o.uu);
                const int k = lane % R0, cls = r + R0 * (lane / R0);
#pragma unroll
                for (int a = 0; a < NV; a++) v[a] = u[xc_at(q + Q * a, lane)];
                if constexpr (HOLD_TW) dft_q<-1, true>(v, w_3, 2 * k >= R0, qt, scr);
                else dft_q<-1, true>(v, o.rot_3(), 2 * k >= R0, qt, scr);
                /* output m: element cls of class k + R0 m */
#pragma unroll
                for (int a = 0; a < NV; a++) {
                    const int c = k + R0 * (q + Q * a);
                    put(tb, o.f, c / Tc, (o.f * CL + o.uk2) * NP + tb_at(cls, c % Tc), v[a]);
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
                    for (int c = 0; c < CL; c++) v += cabs2d(tb[(CL + c) * NP + tb_at(rk * J + j, t2l)]);
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

template <typename R, int F, int M, int CL, int P, int NTHR, int MINB, int Q>
__global__ void __launch_bounds__(NTHR, MINB) wide_kernel(LaunchArgs a)
{
    drive<R, typename Wide<R, F, M, CL, P, NTHR, MINB, Q>::Engine>(a);
}

}  // namespace cuopo
