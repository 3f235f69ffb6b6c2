/*
 * fft.cuh -- register/shared-memory Stockham FFT used inside the fused
 * SSFM kernels.  Replaces the cufftExecC2C calls of the reference
 * (src/headers/cwes2.cuh:170-182, src/headers/cwes3.cuh:175-193,
 * src/cuOPO.cu:522-550): unnormalised C2C, exponent sign S = +1 for
 * CUFFT_INVERSE and S = -1 for CUFFT_FORWARD.
 *
 * Algorithm: Stockham autosort (Cooley-Tukey radix-r stages with the
 * reordering folded into each stage's store), mixed radix: one first
 * stage of radix 2/4/8 when log2(M) is not a multiple of 4, then radix-16
 * stages.  Every thread of the CTA holds E = 16 points of one field in
 * registers; stage outputs go through shared memory to the next stage.
 *
 * Thread t holds points t + e*T (T = M/16 threads, e = 0..15) both before
 * the first stage and after the last one, for any stage plan, so the
 * element-wise work of the solver (RK4, dispersion, cavity map) runs on
 * those registers with no shared-memory exchange or barrier.
 *
 * Twiddles are applied as rotations built from three shears,
 *   x -= t y;  y += s x;  x -= t y,      t = tan(phi/2), s = sin(phi),
 * after an exact quarter-turn step (a multiple of i) that leaves
 * |phi| <= pi/4 (Paeth's three-shear rotation).  Each shear has determinant
 * exactly 1 whatever the float values of t and s, so a rotation never
 * changes the power of a field with random phase to first order; a complex
 * multiplication by float-rounded (cos, sin) does (by |w_f|^2 - 1, a few
 * 1e-8, systematically), and over the ~10^6 transforms of a long cavity run
 * that bias moves the steady-state power by ~1e-4.
 *
 * A radix-16 stage whose sub-transform length is NS needs W^{r k},
 * W = exp(2 pi i/(16 NS)), k = t mod NS, on input r = b + 4a of the 4 x 4
 * transform.  W^{4 a k} depends on a only and W^{b k} on b only, so the
 * first is applied before the inner 4-point transforms over a, and the
 * second after them (they are linear), together with their own W16^{b q}:
 * 12 + 12 rotations and 8 constant ones per 16 points, each input rotated
 * once by each factor.  (Rotating every input by W^{b k} and then a times by
 * W^{4k} took 36 and 8: 132 multiply-adds of the 16-point stage's 276
 * against 96 of 240 here, and up to four roundings in a row against two.)
 * The six angles of a stage are 1, 2, 3 (below 3 pi/8) and 4, 8, 12 (in
 * [0, 3 pi/2)) times 2 pi k/(16 NS); the last two are brought into
 * [-pi/2, pi/2] by a quarter turn that is the same for every k (8) or one of
 * two (12).  The last stage keeps its six angles in registers, middle
 * stages read theirs from a small shared-memory table.
 */
#pragma once
#include "cplx.cuh"

namespace cuopo {

/* x * i^m (exact). */
template <int m, typename C>
__device__ __forceinline__ C iq(C x)
{
    constexpr int q = ((m % 4) + 4) % 4;
    if constexpr (q == 0) return x;
    else if constexpr (q == 1) return mk<C>(-x.y, x.x);
    else if constexpr (q == 2) return mk<C>(-x.x, -x.y);
    else return mk<C>(x.y, -x.x);
}

template <typename C>
__device__ __forceinline__ C iq_rt(C x, int m)
{
    using R = typename real_of<C>::type;
    R a = (m & 1) ? -x.y : x.x;
    R b = (m & 1) ? x.x : x.y;
    if (m & 2) {
        a = -a;
        b = -b;
    }
    return mk<C>(a, b);
}

/* Rotation of x by phi given (t, s) = (tan(phi/2), sin(phi)), three shears. */
template <typename C, typename R>
__device__ __forceinline__ C shear_rot(C x, R t, R s)
{
    const R x1 = rfma(-t, x.y, x.x);
    const R y2 = rfma(s, x1, x.y);
    const R x3 = rfma(-t, y2, x1);
    return mk<C>(x3, y2);
}

/* exp(S * i * pi * K / 8) * x, K compile-time: quarter turns times a
 * rotation by r pi / 8, |r| <= 2. */
template <int S, int K, typename C>
__device__ __forceinline__ C tw16(C x)
{
    using R = typename real_of<C>::type;
    constexpr int n = S * (((K % 16) + 16) % 16);            /* angle n pi / 8 */
    constexpr int m = n >= 0 ? (n + 1) / 4 : -((-n + 1) / 4); /* nearest quarter turn */
    constexpr int r = n - 4 * m;                               /* -1..2 */
    constexpr double T1 = 0.19891236737965800691;              /* tan(pi/16) */
    constexpr double S1 = 0.38268343236508977173;              /* sin(pi/8) */
    constexpr double T2 = 0.41421356237309504880;              /* tan(pi/8) */
    constexpr double S2 = 0.70710678118654752440;              /* sin(pi/4) */
    const C y = iq<m>(x);
    if constexpr (r == 0) return y;
    else if constexpr (r == 1) return shear_rot(y, (R)T1, (R)S1);
    else if constexpr (r == -1) return shear_rot(y, (R)-T1, (R)-S1);
    else if constexpr (r == 2) return shear_rot(y, (R)T2, (R)S2);
    else return shear_rot(y, (R)-T2, (R)-S2);
}

template <int S, typename C>
__device__ __forceinline__ void dft2(C &x0, C &x1)
{
    const C a = cadd(x0, x1), b = csub(x0, x1);
    x0 = a;
    x1 = b;
}

template <int S, typename C>
__device__ __forceinline__ void dft4(C &x0, C &x1, C &x2, C &x3)
{
    const C a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = csub(x1, x3);
    const C sd = cmul_si<S>(d);
    x0 = cadd(a, c);
    x2 = csub(a, c);
    x1 = cadd(b, sd);
    x3 = csub(b, sd);
}

/* 8 = 2 x 4: n = b + 2a, k = q1 + 4 q2. */
template <int S, typename C>
__device__ __forceinline__ void dft8(C (&v)[8])
{
    dft4<S>(v[0], v[2], v[4], v[6]);
    dft4<S>(v[1], v[3], v[5], v[7]);
    v[3] = tw16<S, 2>(v[3]);
    v[5] = tw16<S, 4>(v[5]);
    v[7] = tw16<S, 6>(v[7]);
    C o[8];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        o[q] = cadd(v[2 * q], v[2 * q + 1]);
        o[q + 4] = csub(v[2 * q], v[2 * q + 1]);
    }
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = o[q];
}

/* The six rotations (tan(phi/2), sin(phi)) of one k of a twiddled radix-16
 * stage: phi = j kappa for b[j-1] (j = 1, 2, 3) and, for a[0..2], 4 kappa,
 * 8 kappa - pi/2 and 12 kappa - pi/2 (k < NS/2) or - pi (otherwise),
 * kappa = 2 pi k / (16 NS). */
template <typename C>
struct StageRot {
    C b[3], a[3];
};

/* x rotated by the quarter turns of the factor W^{12 k}: one (hi = 0) or two
 * (hi = 1), in the direction S. */
template <int S, typename C>
__device__ __forceinline__ C iq12(C x, bool hi)
{
    if constexpr (S > 0) return mk<C>(-(hi ? x.x : x.y), hi ? -x.y : x.x);
    else return mk<C>(hi ? -x.x : x.y, -(hi ? x.y : x.x));
}

/* 16 = 4 x 4: n = b + 4a, k = q1 + 4 q2.  TW: the stage's twiddles (StageRot
 * w, hi = k >= NS/2) applied on the way. */
template <int S, bool TW, typename C>
__device__ __forceinline__ void dft16(C (&v)[16], const StageRot<C> &w, bool hi)
{
    using R = typename real_of<C>::type;
    const R sg = (R)S;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        if constexpr (TW) {
            v[b + 4] = shear_rot(v[b + 4], sg * w.a[0].x, sg * w.a[0].y);
            v[b + 8] = shear_rot(iq<S>(v[b + 8]), sg * w.a[1].x, sg * w.a[1].y);
            v[b + 12] = shear_rot(iq12<S>(v[b + 12], hi), sg * w.a[2].x, sg * w.a[2].y);
        }
        dft4<S>(v[b], v[b + 4], v[b + 8], v[b + 12]);
    }
    /* u_b[q1] = v[b + 4 q1] *= W16^{b q1} */
    v[5] = tw16<S, 1>(v[5]);
    v[9] = tw16<S, 2>(v[9]);
    v[13] = tw16<S, 3>(v[13]);
    v[6] = tw16<S, 2>(v[6]);
    v[10] = tw16<S, 4>(v[10]);
    v[14] = tw16<S, 6>(v[14]);
    v[7] = tw16<S, 3>(v[7]);
    v[11] = tw16<S, 6>(v[11]);
    v[15] = tw16<S, 9>(v[15]);
    if constexpr (TW) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int b = 1; b < 4; b++) v[4 * q + b] = shear_rot(v[4 * q + b], sg * w.b[b - 1].x, sg * w.b[b - 1].y);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) dft4<S>(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    /* X[q1 + 4 q2] = v[4 q1 + q2] */
    C o[16];
#pragma unroll
    for (int q1 = 0; q1 < 4; q1++)
#pragma unroll
        for (int q2 = 0; q2 < 4; q2++) o[q1 + 4 * q2] = v[4 * q1 + q2];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = o[q];
}

template <int S, int RADIX, typename C>
__device__ __forceinline__ void dft(C (&v)[RADIX])
{
    if constexpr (RADIX == 2) dft2<S>(v[0], v[1]);
    else if constexpr (RADIX == 4) dft4<S>(v[0], v[1], v[2], v[3]);
    else if constexpr (RADIX == 8) dft8<S>(v);
    else dft16<S, false>(v, StageRot<C>{}, false);
}

/* Shared-memory index swizzle: XOR of the low bits with the row number so
 * that the stride-R stores of early stages hit distinct banks.  Rows are
 * 128 bytes (16 float2 or 8 double2). */
template <typename C>
__device__ __forceinline__ int swz(int i)
{
    if constexpr (sizeof(C) == 8) return i ^ ((i >> 4) & 15);
    else return i ^ ((i >> 3) & 7);
}

/* Stage plan of an M-point transform (M = 2^m, 16 <= M). */
template <int M>
struct StagePlan {
    static constexpr int lg(int x) { return x <= 1 ? 0 : 1 + lg(x / 2); }
    static constexpr int m = lg(M);
    static_assert((1 << m) == M && M >= 16, "M must be a power of 2 >= 16");
    static constexpr int R0 = (m % 4 == 0) ? 16 : (1 << (m % 4));
    static constexpr int P = (m % 4 == 0) ? m / 4 : m / 4 + 1;
    static constexpr int T = M / 16;
    static constexpr int radix(int p) { return p == 0 ? R0 : 16; }
    static constexpr int ns(int p)
    {
        int n = 1;
        for (int q = 0; q < p; q++) n *= radix(q);
        return n;
    }
};

/* Shared-memory table of the middle radix-16 stages 1..P-2: for stage p and
 * k < NS_p the six rotations of StageRot, stored as [p][k][6] (16-byte
 * loads, conflict-free for consecutive k). */
template <int M>
struct TwTable {
    using SP = StagePlan<M>;
    static constexpr int offset(int p)
    {
        int o = 0;
        for (int q = 1; q < p; q++) o += 6 * SP::ns(q);
        return o;
    }
    static constexpr int size() { return SP::P > 2 ? offset(SP::P - 1) : 0; }
};

/* The six rotations of stage length 512, [k][6] (tan, sin), formed in
 * extended precision when the library is built (build.py): those of a shorter
 * stage are every (512/NS)-th row.  A kernel that formed its own (FP64
 * sincospi, 6 per thread and 6 NS per table) spent 5 us of each launch on
 * them. */
static constexpr int TW_NS = 512;
__device__ __align__(16) static const float2 g_tw_f32[6 * TW_NS] = {
#define CUOPO_TW(t, s) {(float)(t), (float)(s)},
#include "twiddle_table.inc"
#undef CUOPO_TW
};
__device__ __align__(16) static const double2 g_tw_f64[6 * TW_NS] = {
#define CUOPO_TW(t, s) {t, s},
#include "twiddle_table.inc"
#undef CUOPO_TW
};

/* Row k of a stage of length ns. */
template <typename C>
__device__ __forceinline__ const C *tw_row(int k, int ns)
{
    const int i = 6 * k * (TW_NS / ns);
    if constexpr (sizeof(C) == 8) return g_tw_f32 + i;
    else return g_tw_f64 + i;
}

/* Fills the table (all threads of the CTA cooperate; caller syncs). */
template <int M, typename C>
__device__ __forceinline__ void fill_twiddle_table(C *tab, int t, int nthreads = StagePlan<M>::T)
{
    using SP = StagePlan<M>;
#pragma unroll
    for (int p = 1; p + 1 < SP::P; p++) {
        const int ns = SP::ns(p);
        const int off = TwTable<M>::offset(p);
        for (int idx = t; idx < 6 * ns; idx += nthreads) tab[off + idx] = tw_row<C>(idx / 6, ns)[idx % 6];
    }
}

/* Six rotations of one table row, as 16-byte loads (rows are 48 or 96 bytes). */
__device__ __forceinline__ StageRot<float2> load_rot(const float2 *row)
{
    const float4 *q = reinterpret_cast<const float4 *>(row);
    const float4 u = q[0], v = q[1], w = q[2];
    StageRot<float2> r;
    r.b[0] = make_float2(u.x, u.y);
    r.b[1] = make_float2(u.z, u.w);
    r.b[2] = make_float2(v.x, v.y);
    r.a[0] = make_float2(v.z, v.w);
    r.a[1] = make_float2(w.x, w.y);
    r.a[2] = make_float2(w.z, w.w);
    return r;
}

__device__ __forceinline__ StageRot<double2> load_rot(const double2 *row)
{
    StageRot<double2> r;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        r.b[j] = row[j];
        r.a[j] = row[3 + j];
    }
    return r;
}

/* Keeps a value loaded from a constant table in registers: without it the
 * compiler loads it again wherever it is used. */
__device__ __forceinline__ void pin(float2 &v) { asm volatile("" : "+f"(v.x), "+f"(v.y)); }
__device__ __forceinline__ void pin(double2 &v) { asm volatile("" : "+d"(v.x), "+d"(v.y)); }

/* The last radix-16 stage's rotations of thread t. */
template <int M, typename C>
struct StageTwiddles {
    StageRot<C> last;
    const C *tab;      /* shared-memory table of the middle stages */
    __device__ __forceinline__ void init(int t, const C *table)
    {
        using SP = StagePlan<M>;
        tab = table;
        if constexpr (SP::P > 1) {
            const int ns = SP::ns(SP::P - 1);
            last = load_rot(tw_row<C>(t % ns, ns));
#pragma unroll
            for (int j = 0; j < 3; j++) {
                pin(last.a[j]);
                pin(last.b[j]);
            }
        }
    }
};

template <int S, int M, int P_IDX, typename C>
__device__ __forceinline__ void stage_compute(C (&reg)[16], const StageTwiddles<M, C> &tw)
{
    using SP = StagePlan<M>;
    constexpr int R = SP::radix(P_IDX);
    constexpr int NS = SP::ns(P_IDX);
    constexpr int B = 16 / R;
#pragma unroll
    for (int b = 0; b < B; b++) {
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = reg[b + r * B];
        if constexpr (NS > 1) {
            static_assert(R == 16, "twiddled stages are radix 16");
            const int k = threadIdx.x % NS;
            if constexpr (P_IDX + 1 == SP::P) dft16<S, true>(v, tw.last, 2 * k >= NS);
            else dft16<S, true>(v, load_rot(tw.tab + TwTable<M>::offset(P_IDX) + 6 * k), 2 * k >= NS);
        } else {
            dft<S, R>(v);
        }
#pragma unroll
        for (int r = 0; r < R; r++) reg[b + r * B] = v[r];
    }
}

/* Stage P_IDX output to shared memory at its Stockham positions. */
template <int M, int P_IDX, typename C>
__device__ __forceinline__ void stage_store(C *buf, const C (&reg)[16], int t)
{
    using SP = StagePlan<M>;
    constexpr int R = SP::radix(P_IDX);
    constexpr int NS = SP::ns(P_IDX);
    constexpr int B = 16 / R;
    constexpr int T = SP::T;
#pragma unroll
    for (int b = 0; b < B; b++) {
        const int j = t + b * T;
        const int k = j % NS;
        const int base = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) buf[swz<C>(base + r * NS)] = reg[b + r * B];
    }
}

template <int M, typename C>
__device__ __forceinline__ void load_own(const C *buf, C (&reg)[16], int t)
{
    constexpr int T = StagePlan<M>::T;
#pragma unroll
    for (int e = 0; e < 16; e++) reg[e] = buf[swz<C>(t + e * T)];
}

template <int M, typename C>
__device__ __forceinline__ void store_own(C *buf, const C (&reg)[16], int t)
{
    constexpr int T = StagePlan<M>::T;
#pragma unroll
    for (int e = 0; e < 16; e++) buf[swz<C>(t + e * T)] = reg[e];
}

/*
 * Local M-point transform of the registers of the CTA (exponent sign S).
 * Exchange x (counted from X0 within the caller's sequence) goes through
 * buffer (x even ? bufA : bufB).  INPLACE: bufA == bufB, and every
 * exchange is bracketed by two barriers instead of one.  `early` runs while
 * the last exchange is under way (its stores are issued, no register holds
 * data): loads issued there have the barrier and the last stage to arrive.
 */
struct NoEarly {
    __device__ __forceinline__ void operator()() const {}
};

template <int S, int M, int X0, bool INPLACE, int P_IDX = 0, typename C, typename Early = NoEarly>
__device__ __forceinline__ void local_transform(C (&reg)[16], C *bufA, C *bufB,
                                                const StageTwiddles<M, C> &tw, int t, const Early &early = Early())
{
    constexpr int P = StagePlan<M>::P;
    stage_compute<S, M, P_IDX>(reg, tw);
    if constexpr (P_IDX + 1 < P) {
        C *buf = ((X0 + P_IDX) % 2 == 0) ? bufA : bufB;
        if constexpr (INPLACE) __syncthreads();
        stage_store<M, P_IDX>(buf, reg, t);
        if constexpr (P_IDX + 2 == P) early();
        __syncthreads();
        load_own<M>(buf, reg, t);
        local_transform<S, M, X0, INPLACE, P_IDX + 1>(reg, bufA, bufB, tw, t, early);
    }
}

/* Loads that stay where they are written; in-place transforms read data
 * that the kernel writes elsewhere, so not through the read-only path. */
__device__ __forceinline__ float2 ld_stream(const float2 *p)
{
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ld_stream(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

/* Read-only loads that stay where they are written (the compiler moves __ldg
 * down to its use when registers are short, and every use then waits). */
__device__ __forceinline__ float2 ld_now(const float2 *p)
{
    float2 v;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ld_now(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

}  // namespace cuopo
