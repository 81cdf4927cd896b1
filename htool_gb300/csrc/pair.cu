// FP64 products on paired panels: both phases of the product as one streaming
// kernel in packed double-float arithmetic.
//
// The FP64 factors are laid out once per H-matrix as panels of at most 32
// outputs x ncol inputs whose entries are already split into (hi, lo) floats
// (split64_near), two neighbouring outputs side by side in 16 bytes:
// {hi0, hi1, lo0, lo1}, an input's ceil(h / 2) pairs contiguous, inputs one
// after the other.
//   phase 1: the outputs are the phase-1 sums of the leaves on one source
//            cluster tile (their Vt columns stacked, 32 at a time), the
//            inputs the tile's rows of x: no sum crosses lanes, whatever the
//            rank and the tile's height
//   phase 2: the outputs are rows of a target cluster, the inputs the columns
//            of every leaf on it (dense columns of x, phase-1 sums)
// so one kernel serves both.  A warp owns a panel: lane = (pair of outputs,
// slice of the inputs), the panel's bytes arrive by bulk copies in a ring of
// shared-memory stages, the inputs' coefficients by 16-byte asynchronous
// copies in the layout the arithmetic wants ({hi of two right-hand sides, lo
// of two}).  Warps claim panels from a ticket, its next value and the next
// panel's descriptor always requested a panel ahead.
//
// Arithmetic: fma / add / sub on float pairs (.f32x2), two right-hand
// sides per instruction (one right-hand side: two outputs per instruction);
// the multiply-add takes 10 instead of the 12 operations of df_fma, as
//   t = s + p, p = RN(uh xh);  s + p = t + w exactly up to the rest
//   l = fma(uh, xh, -(t - s)) = (p - (t - s)) + (uh xh - p)
// gets the rounding errors of the product and of the sum in one operation.
// The FP32 pipe takes 128 lane operations a clock and SM, so a product with
// one right-hand side is bound by HBM, with four and more by that pipe.
//
// Measured against the tile and chunk kernels of stream.cu and
// matvec_kernels.cu (which shuffle every coefficient, reduce every tile over
// the warp and leave lanes idle on tiles of few rows), Laplace sphere, FP64:
//   100 000 points  1 right-hand side 0.485 -> 0.342 ms, 2: 0.82 -> 0.379,
//                   4: 1.81 -> 0.551, 8: 2.66 -> 0.989
//   400 000 points  1: 2.15 -> 1.57 (6.7 TB/s in phase 1, 7.0 in phase 2, a
//                   copy takes 6.8), 4: 8.05 -> 2.42
// at no larger an error against the FP64 pipe, though 35% of phase 2 ran on it
// there (six inputs each; Laplace 1.9e-14 .. 2.3e-14 -> 1.0e-14 .. 1.8e-14,
// Helmholtz 2.6e-14 .. 4.8e-14 -> 2.4e-14 .. 3.1e-14): both operands are rounded
// to 2^-48 here and truncated at 2^-46 there.
//
// Every wait is bounded; a warp whose wait ran out records status 2, lets its
// copies in flight land (again bounded) and ends.
#include "f32x2.cuh"
#include "kernels.hpp"

#include <algorithm>

namespace htgpu {
namespace {

constexpr int kPairWarps = 4; // warps per CTA, each with its own panels and ring

__device__ long long g_pair_skip = -1; // a panel whose first copy is left out (test support)

// a double as hi + lo, both rounded to nearest (|a - hi - lo| <= 2^-48 |a|, and
// 2^-149 below 2^-101, where the floats run into the subnormal ones; the
// truncating split64 of the other kernels keeps 2^-46 and drops what is below
// 2^-103), by bit operations: the conversions between double and float run on
// the FP64 pipe. |a| < 2^126; zero gives 0, a value that is not finite NaN, so
// that it reaches the outputs
__device__ __forceinline__ F2 split64_near(double a) {
    const long long b  = __double_as_longlong(a);
    const int e        = (int)(b >> 52) & 0x7FF;
    const long long m  = b + (1LL << 28);           // hi: 29 bits rounded off
    const unsigned sg  = (unsigned)((unsigned long long)b >> 32) & 0x80000000u;
    const unsigned hb  = (((unsigned)(m >> 29)) - 0xC0000000u) | sg; // exponent 1023 -> 127 (mod 512), 23 fraction bits
    const int r        = (int)(b - (m & ~((1LL << 29) - 1))); // a - hi in units of 2^(e - 1075), |r| <= 2^28
    F2 f;
    const float lo = (__int2float_rn(r) * 9.31322574615478515625e-10f) * __int_as_float((e - 918) << 23); // 2^-30, 2^(e - 1045)
    const bool ok  = (unsigned)(e - 920) < 229u;
    f.hi           = ok ? __uint_as_float(hb) : e == 0x7FF ? __int_as_float(0x7fffffff) : 0.f;
    f.lo           = ok ? __int_as_float(__float_as_int(lo) ^ (int)sg) : 0.f;
    if ((unsigned)(e - 873) < 47u) { // the same, each scaled down by two normal powers of two
        const int eh = (int)(m >> 52) & 0x7FF;
        f.hi = __int_as_float(__float_as_int((__uint_as_float((hb & 0x7FFFFFu) | 0x3F800000u) * 0x1p-64f) * __int_as_float((eh - 832) << 23)) ^ (int)sg);
        f.lo = __int_as_float(__float_as_int((__int2float_rn(r) * 0x1p-94f) * __int_as_float((e - 854) << 23)) ^ (int)sg);
    }
    return f;
}

// Per Q (pairs of right-hand sides; 0: one right-hand side): input columns
// per stage, stages per warp, resident CTAs per SM.  Two long stages and twelve
// warps an SM beat three of 16 columns and sixteen warps (the bookkeeping of a
// stage against 4 or 8 KB of data; 100 000 points, 4 right-hand sides 0.66 ->
// 0.58 ms); 24 columns keep the three CTAs in shared memory with 6 and 8.
template <int Q>
struct PairCfg {
    static constexpr int kCols   = Q >= 3 ? 24 : 32;
    static constexpr int kStages = 2;
    static constexpr int kCtas   = 3;
    static constexpr int kUnit   = Q ? 16 * Q : 8;              // bytes of an input's coefficients
    static constexpr int kData   = 256 * kCols;                 // 16 pairs x 16 bytes a column
    static constexpr int kCoef   = kData;                       // [q][column]
    static constexpr int kDesc   = kCoef + kUnit * kCols;       // int4: h, columns, last chunk of its panel, output base
    static constexpr int kStage  = (kDesc + 16 + 15) & ~15;
    static constexpr int kBar    = kStages * kStage;
    static constexpr int kWarp   = (kBar + 8 * kStages + 127) & ~127;
    static constexpr int kSmem   = kPairWarps * kWarp;
};

template <int Q>
constexpr int kPairAcc = Q ? 2 * Q : 1; // Q = 0: one, its two halves the two outputs; else [output][q]

// one landed chunk (h outputs, nc inputs) into the lane's accumulators
template <int Q>
__device__ __forceinline__ void pair_chunk(const unsigned char *st, int h, int nc, int lane, DF2 (&acc)[kPairAcc<Q>]) {
    using C      = PairCfg<Q>;
    const int hp = (h + 1) >> 1, S = 32 / hp, slice = lane / hp;
    if (slice < S) {
        const float4 *data = reinterpret_cast<const float4 *>(st) + lane - slice * hp;
        if constexpr (Q == 0) {
            const float2 *cf = reinterpret_cast<const float2 *>(st + C::kCoef);
#pragma unroll 4
            for (int t = slice; t < nc; t += S) {
                const float4 u = data[t * hp];
                const float2 x = cf[t];
                df2_fma(acc[0], fx(u.x, u.y), fx(u.z, u.w), fx(x.x, x.x), fx(x.y, x.y));
            }
        } else {
            const float4 *cf = reinterpret_cast<const float4 *>(st + C::kCoef);
#pragma unroll 2
            for (int t = slice; t < nc; t += S) {
                const float4 u = data[t * hp];
                const f2x h0 = fx(u.x, u.x), h1 = fx(u.y, u.y), l0 = fx(u.z, u.z), l1 = fx(u.w, u.w);
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    const float4 x = cf[q * C::kCols + t];
                    const f2x xh = fx(x.x, x.y), xl = fx(x.z, x.w);
                    df2_fma(acc[q], h0, l0, xh, xl);
                    df2_fma(acc[Q + q], h1, l1, xh, xl);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kPairAcc<Q>; i++)
        df2_renorm(acc[i]);
}

// the slices' sums, in order, to the lanes of slice 0
template <int Q>
__device__ __forceinline__ void pair_slices(int h, int lane, DF2 (&acc)[kPairAcc<Q>]) {
    const int hp = (h + 1) >> 1, S = 32 / hp;
    for (int sl = 1; sl < S; sl++) {
#pragma unroll
        for (int i = 0; i < kPairAcc<Q>; i++) {
            const int src = (lane + sl * hp) & 31;
            DF2 o;
            o.s = shfl2(acc[i].s, src);
            o.c = shfl2(acc[i].c, src);
            if (lane < hp)
                acc[i] = df2_add(acc[i], o);
        }
    }
#pragma unroll
    for (int i = 0; i < kPairAcc<Q>; i++)
        df2_renorm(acc[i]);
}

// the sums of the outputs 2 pair, 2 pair + 1 of a panel to A (P1) or z
template <int Q, bool P1>
__device__ __forceinline__ void pair_store(int h, int out, int pair, const DF2 (&acc)[kPairAcc<Q>], const int *__restrict__ oslot, float *__restrict__ A, float2 *__restrict__ z, int zlen, int nrhs) {
#pragma unroll
    for (int o = 0; o < 2; o++) {
        if (2 * pair + o >= h)
            break;
        if constexpr (Q == 0) {
            const float2 vs = fx2(acc[0].s), vc = fx2(acc[0].c);
            (P1 ? reinterpret_cast<float2 *>(A) + oslot[out + 2 * pair + o] : z + out + 2 * pair + o)[0] = o ? make_float2(vs.y, vc.y) : make_float2(vs.x, vc.x);
        } else if constexpr (P1) {
            float4 *A4 = reinterpret_cast<float4 *>(A) + (long long)Q * oslot[out + 2 * pair + o];
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const float2 vs = fx2(acc[o * Q + q].s), vc = fx2(acc[o * Q + q].c);
                A4[q]           = make_float4(vs.x, vs.y, vc.x, vc.y);
            }
        } else {
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const float2 vs = fx2(acc[o * Q + q].s), vc = fx2(acc[o * Q + q].c);
                float2 *zr      = z + (long long)(2 * q) * zlen + out + 2 * pair + o;
                if (2 * q < nrhs)
                    zr[0] = make_float2(vs.x, vc.x);
                if (2 * q + 1 < nrhs)
                    zr[zlen] = make_float2(vs.y, vc.y);
            }
        }
    }
}

// the copies of one chunk: columns jc .. jc + nc of panel p into stage st,
// idx the coefficient index of this lane's column (phase 2)
template <int Q, bool P1>
__device__ __forceinline__ void pair_copies(const PairPanel &p, int jc, int nc, int idx, bool data, unsigned char *st, unsigned long long *bar, const unsigned char *mirror, const float *X,
                                            const float *A, unsigned long long pol, int lane) {
    using C      = PairCfg<Q>;
    const int hp = (p.h + 1) >> 1;
    if (lane == 0 && data)
        ring_copy(st, mirror + p.src + (long long)16 * hp * jc, (unsigned)(16 * hp * nc), bar, pol);
    if (lane < nc) {
        const unsigned char *src;
        if constexpr (P1)
            src = reinterpret_cast<const unsigned char *>(X) + (long long)C::kUnit * (p.coef + jc + lane);
        else
            src = idx >= 0 ? reinterpret_cast<const unsigned char *>(A) + (long long)C::kUnit * idx : reinterpret_cast<const unsigned char *>(X) + (long long)C::kUnit * (~idx);
        if constexpr (Q == 0) {
            copy_async<8>(st + C::kCoef + 8 * lane, src);
        } else {
#pragma unroll
            for (int q = 0; q < Q; q++)
                copy_async<16>(st + C::kCoef + 16 * (q * C::kCols + lane), src + 16 * q);
        }
    }
}

// P1: coefficients are the rows of X from panel.coef on, sums go to the slots
// oslot[panel.out ..] of A; else the coefficients cidx[panel.coef ..] name
// slots of A (>= 0) or rows of X (~row), sums go to the rows panel.out .. of z
template <int Q, bool P1>
__global__ void __launch_bounds__(32 * kPairWarps, PairCfg<Q>::kCtas)
    pair_kernel(const PairPanel *__restrict__ panels, int npanels, int *__restrict__ ticket, const unsigned char *__restrict__ mirror, const int *__restrict__ cidx, const int *__restrict__ oslot,
                const float *__restrict__ X, float *__restrict__ A, float2 *__restrict__ z, int zlen, int nrhs, int *__restrict__ status) {
    using C             = PairCfg<Q>;
    constexpr int kCols = C::kCols, kStages = C::kStages;
    extern __shared__ __align__(128) unsigned char smem[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *wbase    = smem + (size_t)wid * C::kWarp;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(wbase + C::kBar);
    if (lane == 0)
        ring_init(bar, kStages);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    const unsigned long long pol = stream_policy();
    const long long skip         = g_pair_skip;

    // ---- panels: the current one (cur, from column jc on), the next one and
    // the ticket after that (lane 0) in flight; the first two are the warp's
    // own, the ticket counts the ones after every warp's first two
    const int nwarps = gridDim.x * kPairWarps;
    int icur = blockIdx.x * kPairWarps + wid, inxt = icur + nwarps, tk = 0;
    PairPanel cur{}, nxt{};
    if (icur < npanels)
        cur = panels[icur];
    if (inxt < npanels)
        nxt = panels[inxt];
    int jc  = 0; // first column of cur not yet issued
    int idx = 0; // the coefficient index of column jc + lane
    auto load_idx = [&]() {
        if constexpr (!P1)
            idx = (icur < npanels && lane < kCols && jc + lane < cur.ncol) ? __ldg(cidx + cur.coef + jc + lane) : 0;
    };
    load_idx();
    pdl_next();
    pdl_wait(); // X, A and the ticket are the previous kernels'
    if (inxt < npanels && lane == 0)
        tk = 2 * nwarps + atomicAdd(ticket, 1);
    int issued = 0;
    auto issue = [&]() { // the next chunk into stage issued % kStages; an empty copy group when none is left
        if (icur < npanels) {
            const int s       = issued % kStages;
            const int nc      = min(kCols, cur.ncol - jc);
            unsigned char *st = wbase + (size_t)s * C::kStage;
            if (lane == 0)
                *reinterpret_cast<int4 *>(st + C::kDesc) = make_int4(cur.h, nc, jc + nc == cur.ncol, cur.out);
            pair_copies<Q, P1>(cur, jc, nc, idx, !(icur == skip && jc == 0), st, &bar[s], mirror, X, A, pol, lane);
            issued++;
            jc += nc;
            if (jc == cur.ncol) {
                jc   = 0;
                cur  = nxt;
                icur = inxt;
                if (inxt < npanels) {
                    inxt = __shfl_sync(0xffffffffu, tk, 0);
                    if (inxt < npanels) {
                        nxt = panels[inxt];
                        if (lane == 0)
                            tk = 2 * nwarps + atomicAdd(ticket, 1);
                    }
                }
            }
            load_idx();
        }
        copies_commit();
    };

    DF2 acc[kPairAcc<Q>];
#pragma unroll
    for (int i = 0; i < kPairAcc<Q>; i++)
        acc[i].s = acc[i].c = 0ull;

#pragma unroll
    for (int s = 0; s < kStages - 1; s++)
        issue();
    bool ok  = true;
    int done = 0;
    while (done < issued) {
        const int s = done % kStages;
        issue(); // into the stage the previous iteration read
        copies_wait<kStages - 1>();
        if (!warp_wait_phase(&bar[s], (done / kStages) & 1)) {
            ok = false;
            break;
        }
        __syncwarp();
        const unsigned char *st = wbase + (size_t)s * C::kStage;
        const int4 d            = *reinterpret_cast<const int4 *>(st + C::kDesc);
        pair_chunk<Q>(st, d.x, d.y, lane, acc);
        if (d.z) { // the panel's last chunk
            pair_slices<Q>(d.x, lane, acc);
            if (2 * lane < d.x)
                pair_store<Q, P1>(d.x, d.w, lane, acc, oslot, A, z, zlen, nrhs);
#pragma unroll
            for (int i = 0; i < kPairAcc<Q>; i++)
                acc[i].s = acc[i].c = 0ull;
        }
        __syncwarp(); // every lane is done with the stage before it is refilled
        done++;
    }
    copies_wait<0>();
    if (!ok) {
        if (lane == 0)
            atomicExch(status, 2);
        for (int p = done; p < issued; p++) // the copies in flight land before the warp leaves
            if (!warp_wait_phase(&bar[p % kStages], (p / kStages) & 1) && lane == 0)
                atomicExch(status, 3);
    }
}

// The same sums with the four warps of a CTA on one panel: warp w takes the
// chunks w, w + 4, .., its partial sums meet in shared memory, and the warps in
// turn add a panel's four up and write them while the others go on.  For
// products with so few panels that whole warps would wait on a few long ones.
template <bool P1>
__global__ void __launch_bounds__(32 * kPairWarps, PairCfg<0>::kCtas)
    pair_coop_kernel(const PairPanel *__restrict__ panels, int npanels, const unsigned char *__restrict__ mirror, const int *__restrict__ cidx, const int *__restrict__ oslot,
                     const float *__restrict__ X, float *__restrict__ A, float2 *__restrict__ z, int zlen, int nrhs, int *__restrict__ status) {
    constexpr int Q     = 0; // one right-hand side
    using C             = PairCfg<Q>;
    constexpr int kCols = C::kCols, kStages = C::kStages;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ DF2 part[2][kPairWarps][16][kPairAcc<Q>];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *wbase    = smem + (size_t)wid * C::kWarp;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(wbase + C::kBar);
    if (lane == 0)
        ring_init(bar, kStages);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    const unsigned long long pol = stream_policy();
    const long long skip         = g_pair_skip;
    // the next chunk to issue: columns jc .. of panel icur
    int icur = blockIdx.x, jc = wid * kCols, idx = 0, issued = 0;
    PairPanel cur{};
    auto seek = [&]() { // to the first panel from icur on with a chunk for this warp
        while (icur < npanels) {
            cur = panels[icur];
            if (jc < cur.ncol)
                break;
            icur += gridDim.x;
            jc = wid * kCols;
        }
        if constexpr (!P1)
            idx = (icur < npanels && lane < kCols && jc + lane < cur.ncol) ? __ldg(cidx + cur.coef + jc + lane) : 0;
    };
    seek();
    pdl_next();
    pdl_wait(); // X and A are the previous kernels'
    auto issue = [&]() {
        if (icur < npanels) {
            const int s  = issued % kStages;
            const int nc = min(kCols, cur.ncol - jc);
            pair_copies<Q, P1>(cur, jc, nc, idx, !(icur == skip && jc == 0), wbase + (size_t)s * C::kStage, &bar[s], mirror, X, A, pol, lane);
            issued++;
            jc += kPairWarps * kCols;
            if (jc < cur.ncol) {
                if constexpr (!P1)
                    idx = (lane < kCols && jc + lane < cur.ncol) ? __ldg(cidx + cur.coef + jc + lane) : 0;
            } else {
                icur += gridDim.x;
                jc = wid * kCols;
                seek();
            }
        }
        copies_commit();
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; s++)
        issue();
    bool ok  = true;
    int done = 0, turn = 0;
    for (int p = blockIdx.x; p < npanels; p += gridDim.x, turn++) {
        const PairPanel d = panels[p];
        DF2 acc[kPairAcc<Q>];
#pragma unroll
        for (int i = 0; i < kPairAcc<Q>; i++)
            acc[i].s = acc[i].c = 0ull;
        for (int j = wid * kCols; j < d.ncol && ok; j += kPairWarps * kCols) {
            const int s = done % kStages;
            issue();
            copies_wait<kStages - 1>();
            if (!warp_wait_phase(&bar[s], (done / kStages) & 1)) { // the warp goes on to every barrier of the CTA, without its chunks
                ok = false;
                break;
            }
            __syncwarp();
            pair_chunk<Q>(wbase + (size_t)s * C::kStage, d.h, min(kCols, d.ncol - j), lane, acc);
            __syncwarp();
            done++;
        }
        pair_slices<Q>(d.h, lane, acc);
        if (2 * lane < d.h)
#pragma unroll
            for (int i = 0; i < kPairAcc<Q>; i++)
                part[turn & 1][wid][lane][i] = acc[i];
        __syncthreads();
        if ((turn & 3) == wid && 2 * lane < d.h) {
#pragma unroll
            for (int i = 0; i < kPairAcc<Q>; i++) {
                acc[i] = part[turn & 1][0][lane][i];
#pragma unroll
                for (int w = 1; w < kPairWarps; w++)
                    acc[i] = df2_add(acc[i], part[turn & 1][w][lane][i]);
                df2_renorm(acc[i]);
            }
            pair_store<Q, P1>(d.h, d.out, lane, acc, oslot, A, z, zlen, nrhs);
        }
    }
    copies_wait<0>();
    if (!ok) {
        if (lane == 0)
            atomicExch(status, 2);
        for (int p = done; p < issued; p++)
            if (!warp_wait_phase(&bar[p % kStages], (p / kStages) & 1) && lane == 0)
                atomicExch(status, 3);
    }
}

// the gathered input of right-hand sides c0 .. c0 + w (those past mu_src
// zero), split relative to the input's largest exponent (shift = 1023 - it):
// [row][q] of {hi, hi, lo, lo}, w = 1: [row] of (hi, lo); entries e, e + step, ..
__device__ __forceinline__ void pair_gather_rows(const double *__restrict__ x, int ldx, const int *__restrict__ perm, int n, int c0, int w, int mu_src, int shift, float *__restrict__ X, long long e,
                                                 long long step) {
    auto value = [&](int src, int c) {
        F2 r{0.f, 0.f};
        if (c >= mu_src)
            return r;
        const double v = x[(long long)c * ldx + src];
        const int ex   = (int)(((unsigned)__double2hiint(v) >> 20) & 0x7FFu);
        if (ex == 0x7FF)
            return split64_near(v);
        return ex != 0 && ex + shift >= 1 ? split64_near(scale_pow2(v, shift)) : r;
    };
    const int Q           = w == 1 ? 1 : w >> 1;
    const long long total = (long long)n * Q;
    for (; e < total; e += step) {
        const int j = (int)(e / Q), q = (int)(e - (long long)j * Q);
        const int src = perm ? perm[j] : j;
        if (w == 1) {
            const F2 a                          = value(src, c0);
            reinterpret_cast<float2 *>(X)[j] = make_float2(a.hi, a.lo);
        } else {
            const F2 a = value(src, c0 + 2 * q), b = value(src, c0 + 2 * q + 1);
            reinterpret_cast<float4 *>(X)[e] = make_float4(a.hi, b.hi, a.lo, b.lo);
        }
    }
}
// clears the three tickets too
__global__ void pair_gather_kernel(const double *__restrict__ x, int ldx, const int *__restrict__ perm, int n, int c0, int w, int mu_src, const int *__restrict__ xexp, float *__restrict__ X,
                                   int *__restrict__ tickets) {
    pdl_next();
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x < 3)
        tickets[threadIdx.x] = 0;
    pair_gather_rows(x, ldx, perm, n, c0, w, mu_src, 1023 - max(*xexp, 1), X, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

// A small input (of one pass) in one kernel of one CTA: its largest exponent,
// the tickets and the gathered input.  A small product is a chain of kernels of
// 2 to 8 us, and this takes one out: 1 000 points 19.2 -> 16.4 us a product, 3 000
// 26.1 -> 24.6.  Beyond that one CTA takes longer than the launch it saves (4 000
// points with eight loads a thread 26.6 us, with two kernels 25.9).
constexpr int kPrepThreads = 1024, kPrepLoads = 3;
static_assert(kPrepThreads * kPrepLoads == kPairPrepMax, "an input read in one step");
__global__ void __launch_bounds__(kPrepThreads) pair_prep_kernel(const double *__restrict__ x, const int *__restrict__ perm, int n, int w, int mu_src, int *__restrict__ xexp, float *__restrict__ X,
                                                                 int *__restrict__ tickets) {
    __shared__ int sm[kPrepThreads / 32];
    pdl_next();
    if (threadIdx.x < 3)
        tickets[threadIdx.x] = 0;
    const int total = n * mu_src;
    int ex[kPrepLoads], m = 0;
#pragma unroll
    for (int k = 0; k < kPrepLoads; k++) {
        const int e = (int)threadIdx.x + kPrepThreads * k;
        ex[k]       = e < total ? (int)(((unsigned)__double2hiint(x[e]) >> 20) & 0x7FFu) : 0;
    }
#pragma unroll
    for (int k = 0; k < kPrepLoads; k++)
        m = max(m, ex[k] == 0x7FF ? 0 : ex[k]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0)
        sm[threadIdx.x >> 5] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, sm[threadIdx.x & 31]);
    if (threadIdx.x == 0)
        *xexp = m;
    pair_gather_rows(x, n, perm, n, 0, w, mu_src, 1023 - max(m, 1), X, threadIdx.x, kPrepThreads);
}

// the tiles' sums of every multi-tile leaf into the first tile's slots
__global__ void pair_reduce_kernel(const LrLeaf *__restrict__ lr, const int *__restrict__ multi, int w, float *__restrict__ A) {
    const LrLeaf L = lr[multi[blockIdx.x]];
    pdl_next();
    pdl_wait();
    if (w == 1) {
        float2 *base = reinterpret_cast<float2 *>(A) + L.a_off;
        for (int e = threadIdx.x; e < L.r; e += blockDim.x) {
            DF a{base[e].x, base[e].y};
#pragma unroll 8
            for (int ch = 1; ch < L.nch; ch++) {
                const float2 v = base[(long long)ch * L.r + e];
                a              = df_add(a, DF{v.x, v.y});
                df_renorm(a);
            }
            base[e] = make_float2(a.s, a.c);
        }
        return;
    }
    const int Q  = w >> 1;
    float4 *base = reinterpret_cast<float4 *>(A) + L.a_off * Q;
    for (int e = threadIdx.x; e < L.r * Q; e += blockDim.x) {
        const float4 v = base[e];
        DF2 a{fx(v.x, v.y), fx(v.z, v.w)};
#pragma unroll 8
        for (int ch = 1; ch < L.nch; ch++) {
            const float4 u = base[(long long)ch * L.r * Q + e];
            a              = df2_add(a, DF2{fx(u.x, u.y), fx(u.z, u.w)});
            df2_renorm(a);
        }
        const float2 s = fx2(a.s), c = fx2(a.c);
        base[e] = make_float4(s.x, s.y, c.x, c.y);
    }
}

// native complex layout: i times the sums (re, im) of every slot pair
__global__ void pair_rotate_kernel(const int2 *__restrict__ rows, long long nrows, int Q, float4 *__restrict__ A) {
    const long long total = nrows * Q;
    pdl_next();
    pdl_wait();
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int2 p               = rows[e / Q];
        const int q                = (int)(e % Q);
        const float4 v             = A[(long long)p.x * Q + q];
        A[(long long)p.y * Q + q] = make_float4(-v.y, v.x, -v.w, v.z);
    }
}

// y[c * ldy + perm[i]] (no perm: i - shift) = sum over the covering clusters
// (largest first) of z, brought back to the input's scale
__global__ void pair_zsum_kernel(const ZItem *__restrict__ items, int nitems, const int *__restrict__ zl, const float2 *__restrict__ z, int zlen, int mu, const int *__restrict__ perm,
                                 const int *__restrict__ xexp, double *__restrict__ y, int ldy, int shift, StatusNote note) {
    const int w    = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    pdl_next();
    if (w >= nitems)
        return;
    const ZItem it = items[w];
    // the atom's z bases, one per lane (more than 32 covering clusters: read again)
    const int nl = it.lend - it.lbeg, base = lane < nl ? zl[it.lbeg + lane] : 0;
    pdl_wait();
    if (note.host && blockIdx.x == 0 && threadIdx.x == 0)
        *note.host = *note.status;
    const int xs = max(*xexp, 1) - 1023;
    const int n  = it.h * mu;
    for (int e0 = 0; e0 < n; e0 += 32) {
        const int e = min(e0 + lane, n - 1), c = e / it.h, i = it.row0 + e - c * it.h;
        const float2 *zc = z + (long long)c * zlen + i;
        DF a{0.f, 0.f};
#pragma unroll 8
        for (int l = 0; l < min(nl, 32); l++) {
            const float2 v = zc[__shfl_sync(0xffffffffu, base, l)];
            a              = df_add(a, DF{v.x, v.y});
            df_renorm(a);
        }
        for (int l = it.lbeg + 32; l < it.lend; l++) {
            const float2 v = zc[zl[l]];
            a              = df_add(a, DF{v.x, v.y});
            df_renorm(a);
        }
        const double v = df_to_double(a);
        // an infinity or NaN has no room in its exponent field, and what has none after the scaling is infinite
        const int ex   = (int)(((unsigned)__double2hiint(v) >> 20) & 0x7FFu);
        const double o = ex == 0x7FF ? v : ex + xs < 0x7FF ? scale_pow2_safe(v, xs) : copysign(__longlong_as_double(0x7FFll << 52), v);
        if (e0 + lane < n)
            y[(long long)c * ldy + (perm ? perm[i] : i - shift)] = o;
    }
}

// ---- layout -----------------------------------------------------------------
// phase 2: lane = output row of the panel; its FP64 row sits in one of the
// target cluster's row-chunk panels (pan0 .. of m rows in all)
__global__ void pair_pack2_kernel(const PairPanel *__restrict__ panels, const PairSource *__restrict__ srcs, int npanels, const PanelItem *__restrict__ pan, const double *__restrict__ fac,
                                  unsigned char *__restrict__ mirror) {
    // a CTA per panel, its warps on slabs of 32 inputs
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int p = blockIdx.x; p < npanels; p += gridDim.x) {
        const PairPanel d  = panels[p];
        const PairSource s = srcs[p];
        const int hp       = (d.h + 1) >> 1;
        if (lane >= 2 * hp)
            continue;
        const bool live = lane < d.h;
        const long long i = s.lo + (live ? lane : 0), nchunk = (s.m + 31) / 32;
        const long long q = ((i + 1) * nchunk - 1) / s.m; // the row chunk of row i: floor(m q / nchunk) <= i
        const PanelItem pi = pan[s.pan0 + q];
        const double *row  = fac + pi.off + (i - (long long)s.m * q / nchunk);
        float *dst         = reinterpret_cast<float *>(mirror + d.src) + 4 * (lane >> 1) + (lane & 1);
        for (int k0 = 32 * (threadIdx.x >> 5); k0 < d.ncol; k0 += 32 * nw)
#pragma unroll 8
            for (int k = k0; k < min(k0 + 32, d.ncol); k++) {
                const F2 f            = split64_near(live ? row[(long long)pi.h * k] : 0.);
                dst[4LL * hp * k]     = f.hi;
                dst[4LL * hp * k + 2] = f.lo;
            }
    }
}

// phase 1: outputs osrc[out ..] (FP64 element offsets of their columns),
// inputs the column's rows; 32 x 32 tiles turned over in shared memory
__global__ void __launch_bounds__(128) pair_pack1_kernel(const PairPanel *__restrict__ panels, int npanels, const long long *__restrict__ osrc, const double *__restrict__ fac,
                                                         unsigned char *__restrict__ mirror) {
    __shared__ float2 tile[4][32][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int p = blockIdx.x; p < npanels; p += gridDim.x) {
        const PairPanel d       = panels[p];
        const int hp            = (d.h + 1) >> 1;
        const long long my_src = lane < d.h ? osrc[d.out + lane] : 0;
        for (int k0 = 32 * wid; k0 < d.ncol; k0 += 128) {
            const int nk = min(32, d.ncol - k0);
            __syncwarp();
#pragma unroll 8
            for (int o = 0; o < 32; o++) {
                const long long so = __shfl_sync(0xffffffffu, my_src, o);
                const F2 f         = split64_near(o < d.h && lane < nk ? fac[so + k0 + lane] : 0.);
                tile[wid][lane][o] = make_float2(f.hi, f.lo);
            }
            __syncwarp();
            if (lane < 2 * hp) {
                float *dst = reinterpret_cast<float *>(mirror + d.src) + 4LL * hp * k0 + 4 * (lane >> 1) + (lane & 1);
                for (int k = 0; k < nk; k++) {
                    const float2 f        = tile[wid][k][lane];
                    dst[4LL * hp * k]     = f.x;
                    dst[4LL * hp * k + 2] = f.y;
                }
            }
        }
    }
}

int pair_sms() {
    int dev = 0, sms = 0;
    HTGPU_CUDA(cudaGetDevice(&dev));
    HTGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max(sms, 1);
}

template <int Q, bool P1>
void launch_pair_q(const PairPanel *panels, int npanels, int *ticket, const unsigned char *mirror, const int *cidx, const int *oslot, const float *X, float *A, float2 *z, int zlen, int nrhs,
                   int *status, cudaStream_t st) {
    static unsigned long long done = 0; // devices whose shared-memory limit was raised
    int dev = 0;
    HTGPU_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !(done >> dev & 1)) {
        HTGPU_CUDA(cudaFuncSetAttribute(pair_kernel<Q, P1>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<Q>::kSmem));
        if (dev < 64)
            done |= 1ull << dev;
    }
    const int resident = PairCfg<Q>::kCtas * pair_sms();
    // one right-hand side and fewer than two panels a CTA: four warps to a
    // panel (4 000 points 0.055 -> 0.046 ms a product; no gain from 10 000 points
    // or with more right-hand sides, whose panels take the warps longer)
    if constexpr (Q == 0)
        if (npanels < 2 * resident) {
            static unsigned long long donec = 0;
            if (dev >= 64 || !(donec >> dev & 1)) {
                HTGPU_CUDA(cudaFuncSetAttribute(pair_coop_kernel<P1>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<0>::kSmem));
                if (dev < 64)
                    donec |= 1ull << dev;
            }
            pdl_launch(pair_coop_kernel<P1>, std::min(resident, npanels), 32 * kPairWarps, PairCfg<0>::kSmem, st, panels, npanels, mirror, cidx, oslot, X, A, z, zlen, nrhs, status);
            return;
        }
    const int nctas = std::min(resident, (npanels + kPairWarps - 1) / kPairWarps);
    pdl_launch(pair_kernel<Q, P1>, nctas, 32 * kPairWarps, PairCfg<Q>::kSmem, st, panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status);
}

template <bool P1>
void launch_pair(const PairPanel *panels, int npanels, int *ticket, const unsigned char *mirror, const int *cidx, const int *oslot, const float *X, float *A, float2 *z, int zlen, int w, int nrhs,
                 int *status, cudaStream_t st) {
    if (npanels <= 0)
        return;
    switch (w) {
    case 1: launch_pair_q<0, P1>(panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status, st); break;
    case 2: launch_pair_q<1, P1>(panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status, st); break;
    case 4: launch_pair_q<2, P1>(panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status, st); break;
    case 6: launch_pair_q<3, P1>(panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status, st); break;
    case 8: launch_pair_q<4, P1>(panels, npanels, ticket, mirror, cidx, oslot, X, A, z, zlen, nrhs, status, st); break;
    default: require(false, "paired panels: 1, 2, 4, 6 or 8 right-hand sides a pass"); break;
    }
}

} // namespace

int pair_pass_width(int left, bool exact) {
    if (left >= 8)
        return 8;
    if (left == 1)
        return 1;
    return (left & 1) && exact ? left - 1 : (left + 1) & ~1;
}

void launch_pair_gather(const double *x, int ldx, const int *perm, int n, int c0, int w, int mu_src, const int *xexp, float *X, int *tickets, cudaStream_t st) {
    const long long total = (long long)n * (w == 1 ? 1 : w >> 1);
    const int blocks      = (int)std::max<long long>(1, std::min<long long>((total + 255) / 256, 16LL * pair_sms()));
    pdl_launch(pair_gather_kernel, blocks, 256, 0, st, x, ldx, perm, n, c0, w, mu_src, xexp, X, tickets);
}

void launch_pair_prep(const double *x, const int *perm, int n, int w, int mu_src, int *xexp, float *X, int *tickets, cudaStream_t st) {
    pair_prep_kernel<<<1, kPrepThreads, 0, st>>>(x, perm, n, w, mu_src, xexp, X, tickets);
    HTGPU_CUDA(cudaGetLastError());
}

void launch_pair_phase1(const PairPanel *panels, int npanels, int *tickets, const unsigned char *mirror, const int *oslot, const float *X, float *A, int w, int *status, cudaStream_t st) {
    launch_pair<true>(panels, npanels, tickets, mirror, nullptr, oslot, X, A, nullptr, 0, w, w, status, st);
}

void launch_pair_phase2(const PairPanel *panels, int npanels, int *tickets, const unsigned char *mirror, const int *cidx, const float *X, float *A, int w, int nrhs, float2 *z, int zlen, int *status,
                        cudaStream_t st) {
    launch_pair<false>(panels, npanels, tickets + 1, mirror, cidx, nullptr, X, A, z, zlen, w, nrhs, status, st);
}

void launch_pair_reduce(const LrLeaf *lr, const int *multi, int nmulti, int w, float *A, cudaStream_t st) {
    if (nmulti <= 0)
        return;
    pdl_launch(pair_reduce_kernel, nmulti, 128, 0, st, lr, multi, w, A);
}

void launch_pair_rotate(const int2 *rows, long long nrows, int w, float *A, cudaStream_t st) {
    require(w >= 2, "complex sums come in pairs of right-hand sides");
    const long long total = nrows * (w >> 1);
    if (total <= 0)
        return;
    pdl_launch(pair_rotate_kernel, (int)std::min<long long>((total + 255) / 256, 4096), 256, 0, st, rows, nrows, w >> 1, reinterpret_cast<float4 *>(A));
}

void launch_pair_zsum(const ZItem *items, int nitems, const int *zl, const float2 *z, int zlen, int mu, const int *perm, const int *xexp, double *y, int ldy, cudaStream_t st, int shift, StatusNote note) {
    if (nitems <= 0)
        return;
    pdl_launch(pair_zsum_kernel, (nitems + 7) / 8, 256, 0, st, items, nitems, zl, z, zlen, mu, perm, xexp, y, ldy, shift, note);
}

void launch_pair_pack(const PairPanel *p1, int np1, const long long *osrc, const PairPanel *p2, const PairSource *s2, int np2, const PanelItem *pan, const double *fac, unsigned char *mirror,
                      cudaStream_t st) {
    const int most = 16 * pair_sms();
    if (np1 > 0)
        pair_pack1_kernel<<<std::min(most, np1), 128, 0, st>>>(p1, np1, osrc, fac, mirror);
    if (np2 > 0)
        pair_pack2_kernel<<<std::min(most, np2), 128, 0, st>>>(p2, s2, np2, pan, fac, mirror);
    HTGPU_CUDA(cudaGetLastError());
}

void set_pair_waits(long long cycles, long long skip) {
    HTGPU_CUDA(cudaMemcpyToSymbol(g_wait_limit, &cycles, sizeof(cycles)));
    HTGPU_CUDA(cudaMemcpyToSymbol(g_pair_skip, &skip, sizeof(skip)));
    set_red_waits(cycles);
}

} // namespace htgpu
