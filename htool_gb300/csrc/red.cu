// Reduced-precision products off the tensor cores on warp-fed streams: the
// FP32 and BF16 columns of the low-rank leaves, both phases, for 1 to 8 right-
// hand sides a pass (their dense FP64 blocks run on paired panels, pair.cu).
//
//   red1_kernel  phase 1 of products with 3 or more right-hand sides.  The Vt
//                columns of the leaves on one source tile are stacked by
//                element kind into panels of at most 64 outputs, the panel's
//                rows (the tile's x rows) one after the other: lane = two
//                outputs, which it sums over the rows in order
//   red2_kernel  phase 2: the chunks of every row chunk in the lane order they
//                are stored in (kernels.hpp, SwizzleJob); lane = (row, slice)
//
// A warp feeds itself as in pair.cu: panels or ranges of chunks claimed from a
// ticket a unit ahead, bytes by bulk copies into a ring of stages,
// coefficients by asynchronous copies right-hand sides side by side, so one
// FMA on a float pair (fma.f32x2, each half rounded like the scalar one) takes
// two right-hand sides, or with one right-hand side two columns.  The FP32 sums
// and their order are those of phase1_stack_kernel and of the chunk kernels in
// stream.cu, which a caller's choice of mode keeps.
//
// Bound by latency (20 warps an SM, in phase 2 with 6 and 8 right-hand sides 12;
// reading half the coefficients, two rows a lane, gained 1%), so descriptors and
// indices are loaded ahead and a row chunk starts from its dense part.  Measured
// against those kernels, Laplace sphere, FP32/BF16 factors, ms a product:
// 100 000 points 1 right-hand side 0.258 -> 0.221, 2: 0.362 -> 0.268, 4: 0.720 ->
// 0.297, 8: 1.82 -> 0.418; 200 000 points 1: 0.505 -> 0.460, 8: 3.66 -> 0.799.
// Every wait is bounded (status 2).
#include "f32x2.cuh"
#include "kernels.hpp"

#include <algorithm>
#include <type_traits>

namespace htgpu {
namespace {

constexpr int kRedWarps  = 4; // warps per CTA, each with its own ring
// Stages per warp.  Twenty warps an SM with one stage on its way each beat
// twelve or sixteen with two (ms of 200 000 points, 3 stages and what then fits
// against this: 1 right-hand side 0.508 -> 0.469, 2: 0.601 -> 0.533, 4: 0.636 ->
// 0.55, 8: 0.904 -> 0.81); 6 and 8 right-hand sides keep 12 warps in phase 2,
// where 16 or 20 leave too few registers (0.52 and more against 0.50 ms).
constexpr int kRedStages = 2;

// floor(t / d) for 0 <= t < 128, 1 <= d <= 32 (exact: the product overshoots
// t / d by less than 128 / 65536, below the 1 / d gap to the next integer)
struct RedRcp {
    unsigned v[33];
};
constexpr RedRcp red_rcp() {
    RedRcp t{};
    for (int d = 1; d <= 32; d++)
        t.v[d] = 65536u / (unsigned)d + 1u;
    return t;
}
__constant__ RedRcp kRedRcp = red_rcp();
__device__ __forceinline__ int red_div(int t, int d) { return (int)(((unsigned)t * kRedRcp.v[d]) >> 16); }

// a chunk's shape in one word: rows (6 bits), columns (7), FP32, flags (5), the
// end of its last column group (8)
__device__ __forceinline__ int red_pack(const StreamChunk &c) { return c.h | c.ncol << 6 | (c.kind == kStreamF32 ? 1 << 13 : 0) | (int)c.flags << 14 | (int)c.pad << 19; }
__device__ __forceinline__ int red_h(int m) { return m & 63; }
__device__ __forceinline__ int red_ncol(int m) { return (m >> 6) & 127; }
__device__ __forceinline__ bool red_f32(int m) { return m >> 13 & 1; }
__device__ __forceinline__ int red_flags(int m) { return (m >> 14) & 31; }
__device__ __forceinline__ int red_end(int m) { return (m >> 19) & 255; }

// one float global -> shared, or zero (nothing is read)
__device__ __forceinline__ void copy_or_zero(float *dst, const float *src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sa(dst)), "l"(src), "r"(live ? 4 : 0) : "memory");
}

// W floats (one row or slot) global -> shared, W x 4-byte aligned
template <int W>
__device__ __forceinline__ void copy_row(float *dst, const float *src) {
    constexpr int B = W % 4 == 0 ? 16 : W % 2 == 0 ? 8 : 4;
#pragma unroll
    for (int i = 0; i < 4 * W; i += B)
        copy_async<B>(reinterpret_cast<unsigned char *>(dst) + i, reinterpret_cast<const unsigned char *>(src) + i);
}

// the W / 2 pairs of right-hand sides of one row in shared memory
template <int W>
__device__ __forceinline__ void load_pairs(const float *p, f2x (&x)[W / 2]) {
    if constexpr (W % 4 == 0) {
#pragma unroll
        for (int q = 0; q < W / 4; q++) {
            const float4 v = reinterpret_cast<const float4 *>(p)[q];
            x[2 * q]       = fx(v.x, v.y);
            x[2 * q + 1]   = fx(v.z, v.w);
        }
    } else {
#pragma unroll
        for (int q = 0; q < W / 2; q++) {
            const float2 v = reinterpret_cast<const float2 *>(p)[q];
            x[q]           = fx(v.x, v.y);
        }
    }
}

// a DF accumulator pair takes two FP32 sums (TwoSum)
__device__ __forceinline__ void df2_addf(DF2 &a, f2x p) {
    const f2x s  = fx_add(a.s, p);
    const f2x bp = fx_sub(s, a.s);
    const f2x e  = fx_add(fx_sub(a.s, fx_sub(s, bp)), fx_sub(p, bp));
    a.s          = s;
    a.c          = fx_add(a.c, e);
}

// ---- phase 1 ----------------------------------------------------------------
template <int W>
struct Red1Cfg {
    static constexpr int kRows  = 32;                      // x rows of a stage at most
    static constexpr int kData  = 4096;
    static constexpr int kDesc  = kData + 4 * W * kRows;    // the data, X
    static constexpr int kStage = (kDesc + 16 + 15) & ~15;
    static constexpr int kBar   = kRedStages * kStage;
    static constexpr int kWarp  = (kBar + 8 * kRedStages + 127) & ~127;
    static constexpr int kSmem  = kRedWarps * kWarp;
    static constexpr int kCtas  = 5;
};

template <int W>
__global__ void __launch_bounds__(32 * kRedWarps, Red1Cfg<W>::kCtas)
    red1_kernel(const RedPanel *__restrict__ panels, int npanels, int *__restrict__ ticket, const unsigned char *__restrict__ mirror, const int2 *__restrict__ outs, const float *__restrict__ scale,
                const float *__restrict__ X, float *__restrict__ A, int *__restrict__ status) {
    using C = Red1Cfg<W>;
    constexpr int Q = W > 1 ? W / 2 : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *wbase    = smem + (size_t)wid * C::kWarp;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(wbase + C::kBar);
    if (lane == 0)
        ring_init(bar, kRedStages);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    const unsigned long long pol = stream_policy();
    const int nwarps             = gridDim.x * kRedWarps;
    int icur = blockIdx.x * kRedWarps + wid, inxt = icur + nwarps, tk = 0;
    RedPanel cur{}, nxt{};
    if (icur < npanels)
        cur = panels[icur];
    if (inxt < npanels)
        nxt = panels[inxt];
    pdl_next();
    pdl_wait(); // X and the ticket are the previous kernels'
    if (inxt < npanels && lane == 0)
        tk = 2 * nwarps + atomicAdd(ticket, 1);
    int jc = 0, issued = 0;
    auto issue = [&]() {
        if (icur < npanels) {
            const int s      = issued % kRedStages;
            const int stride = cur.kind == kStreamF32 ? 16 * ((cur.h + 3) >> 2) : 16 * ((cur.h + 7) >> 3);
            const int nr     = min(min(C::kRows, C::kData / stride), cur.nk - jc);
            unsigned char *st = wbase + (size_t)s * C::kStage;
            if (lane == 0) {
                *reinterpret_cast<int4 *>(st + C::kDesc) = make_int4(cur.h | cur.kind << 8, nr, jc + nr == cur.nk, cur.out);
                ring_copy(st, mirror + cur.src + (long long)stride * jc, (unsigned)(stride * nr), &bar[s], pol);
            }
            if (lane < nr)
                copy_row<W>(reinterpret_cast<float *>(st + C::kData) + W * lane, X + (long long)W * (cur.xrow + jc + lane));
            issued++;
            jc += nr;
            if (jc == cur.nk) {
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
        }
        copies_commit();
    };
    f2x acc[2][Q]; // W = 1: one pair, its halves the two outputs
#pragma unroll
    for (int q = 0; q < Q; q++)
        acc[0][q] = acc[1][q] = 0ull;
#pragma unroll
    for (int s = 0; s < kRedStages - 1; s++)
        issue();
    bool ok  = true;
    int done = 0;
    while (done < issued) {
        const int s = done % kRedStages;
        issue();
        copies_wait<kRedStages - 1>();
        if (!warp_wait_phase(&bar[s], (done / kRedStages) & 1)) {
            ok = false;
            break;
        }
        __syncwarp();
        const unsigned char *st = wbase + (size_t)s * C::kStage;
        const int4 d            = *reinterpret_cast<const int4 *>(st + C::kDesc);
        const int h = d.x & 255, nr = d.y;
        const float *xr = reinterpret_cast<const float *>(st + C::kData);
        if (2 * lane < h) {
            auto rows = [&](auto fp32) {
                constexpr bool F = decltype(fp32)::value;
                const int stride = F ? 16 * ((h + 3) >> 2) : 16 * ((h + 7) >> 3);
                const unsigned char *p = st + (F ? 8 : 4) * lane;
#pragma unroll 4
                for (int j = 0; j < nr; j++, p += stride) {
                    float e0, e1;
                    if constexpr (F) {
                        const float2 v = *reinterpret_cast<const float2 *>(p);
                        e0 = v.x, e1 = v.y;
                    } else {
                        const unsigned v = *reinterpret_cast<const unsigned *>(p);
                        e0 = __uint_as_float(v << 16), e1 = __uint_as_float(v & 0xffff0000u);
                    }
                    if constexpr (W == 1) {
                        const float x = xr[j];
                        acc[0][0]     = fx_fma(fx(e0, e1), fx(x, x), acc[0][0]);
                    } else {
                        f2x x[Q];
                        load_pairs<W>(xr + W * j, x);
#pragma unroll
                        for (int q = 0; q < Q; q++) {
                            acc[0][q] = fx_fma(fx(e0, e0), x[q], acc[0][q]);
                            acc[1][q] = fx_fma(fx(e1, e1), x[q], acc[1][q]);
                        }
                    }
                }
            };
            if ((d.x >> 8) == kStreamF32)
                rows(std::true_type{});
            else
                rows(std::false_type{});
            if (d.z) {
#pragma unroll
                for (int o = 0; o < 2; o++)
                    if (2 * lane + o < h) {
                        const int2 io  = outs[d.w + 2 * lane + o]; // slot, scale index
                        const float sc = __ldg(scale + io.y);
                        float *dst     = A + (long long)W * io.x;
                        if constexpr (W == 1) {
                            const float2 v = fx2(acc[0][0]);
                            dst[0]         = (o ? v.y : v.x) * sc;
                        } else {
#pragma unroll
                            for (int q = 0; q < Q; q++) {
                                const float2 v                      = fx2(acc[o][q]);
                                reinterpret_cast<float2 *>(dst)[q] = make_float2(v.x * sc, v.y * sc);
                            }
                        }
                    }
#pragma unroll
                for (int q = 0; q < Q; q++)
                    acc[0][q] = acc[1][q] = 0ull;
            }
        }
        __syncwarp();
        done++;
    }
    copies_wait<0>();
    if (!ok) {
        if (lane == 0)
            atomicExch(status, 2);
        for (int p = done; p < issued; p++)
            if (!warp_wait_phase(&bar[p % kRedStages], (p / kRedStages) & 1) && lane == 0)
                atomicExch(status, 3);
    }
}

// ---- phase 2 ----------------------------------------------------------------
template <int W>
struct Red2Cfg {
    static constexpr int kCoef  = kStreamStage;                                       // [column][W], W = 1: in lane order
    static constexpr int kDesc  = kCoef + (W == 1 ? 4 * 128 : 4 * W * kStreamCols);
    static constexpr int kStage = (kDesc + 16 + 15) & ~15;
    static constexpr int kBar   = kRedStages * kStage;
    static constexpr int kWarp  = (kBar + 8 * kRedStages + 127) & ~127;
    static constexpr int kSmem  = kRedWarps * kWarp;
    static constexpr int kCtas  = W <= 4 ? 5 : 3;
};

template <int W>
__global__ void __launch_bounds__(32 * kRedWarps, Red2Cfg<W>::kCtas)
    red2_kernel(const StreamChunk *__restrict__ chunks, const int *__restrict__ rbeg, int nranges, int *__restrict__ ticket, const unsigned char *__restrict__ mix, const int *__restrict__ cidx,
                const float *__restrict__ A, float2 *__restrict__ z, int zlen, int nrhs, int *__restrict__ status) {
    using C = Red2Cfg<W>;
    constexpr int Q = W > 1 ? W / 2 : 1;
    extern __shared__ __align__(128) unsigned char smem[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *wbase    = smem + (size_t)wid * C::kWarp;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(wbase + C::kBar);
    if (lane == 0)
        ring_init(bar, kRedStages);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    const unsigned long long pol = stream_policy();
    // ranges of whole row chunks: what is left of the one being taken [k, e),
    // the next one's bounds, the ticket after that.  Their descriptors come 32
    // at a time, one to a lane, a window ahead of their use, and a chunk's
    // column indices two chunks ahead (loaded chunk by chunk, a descriptor and
    // then its indices, they held a warp up for memory latencies)
    const int nwarps = gridDim.x * kRedWarps;
    int icur = blockIdx.x * kRedWarps + wid, inxt = icur + nwarps, tk = 0;
    int k = 0, e = 0, nk = 0, ne = 0;
    if (icur < nranges) {
        k = rbeg[icur];
        e = rbeg[icur + 1];
    }
    if (inxt < nranges) {
        nk = rbeg[inxt];
        ne = rbeg[inxt + 1];
    }
    struct Win {
        long long src;
        int a, b, m, bytes, n;
    };
    auto load_window = [&](Win &w) {
        w.n = min(32, e - k);
        if (lane < w.n) {
            const StreamChunk c = chunks[k + lane];
            w.src               = c.src;
            w.a                 = c.a;
            w.b                 = c.b;
            w.bytes             = c.bytes;
            w.m                 = red_pack(c);
        }
        k += w.n;
    };
    Win w0{}, w1{};
    load_window(w0);
    pdl_next();
    pdl_wait(); // A, z and the ticket are the previous kernels'
    if (inxt < nranges && lane == 0)
        tk = 2 * nwarps + atomicAdd(ticket, 1);
    auto next_window = [&]() {
        if (k >= e && inxt < nranges) {
            k    = nk;
            e    = ne;
            inxt = __shfl_sync(0xffffffffu, tk, 0);
            if (inxt < nranges) {
                nk = rbeg[inxt];
                ne = rbeg[inxt + 1];
                if (lane == 0)
                    tk = 2 * nwarps + atomicAdd(ticket, 1);
            }
        }
        load_window(w1); // empty past the last range
    };
    next_window();
    struct Chunk {
        long long src;
        int b, m, bytes, ix0, ix1;
    };
    int at          = 0;
    auto next_chunk = [&]() { // m = 0: no more
        Chunk c{};
        if (at == w0.n) {
            w0 = w1;
            at = 0;
            if (w0.n > 0)
                next_window();
        }
        if (w0.n > 0) {
            c.src       = __shfl_sync(0xffffffffu, w0.src, at);
            c.b         = __shfl_sync(0xffffffffu, w0.b, at);
            c.m         = __shfl_sync(0xffffffffu, w0.m, at);
            c.bytes     = __shfl_sync(0xffffffffu, w0.bytes, at);
            const int a = __shfl_sync(0xffffffffu, w0.a, at), n = red_ncol(c.m);
            c.ix0 = lane < n ? __ldg(cidx + a + lane) : 0;
            c.ix1 = lane + 32 < n ? __ldg(cidx + a + lane + 32) : 0;
            at++;
        }
        return c;
    };
    Chunk d0 = next_chunk(), d1 = next_chunk();
    int issued = 0;
    auto issue = [&]() {
        if (d0.m != 0) {
            const int s = issued % kRedStages, ncol = red_ncol(d0.m), end = red_end(d0.m);
            unsigned char *st = wbase + (size_t)s * C::kStage;
            float *cf         = reinterpret_cast<float *>(st + C::kCoef);
            if (lane == 0) {
                *reinterpret_cast<int2 *>(st + C::kDesc) = make_int2(d0.m, d0.b);
                ring_copy(st, mix + d0.src, (unsigned)d0.bytes, &bar[s], pol);
            }
            // past the chunk's columns, up to the last group's end, the data are
            // zero; the coefficients there must be numbers (the stage's last
            // chunk may have left a NaN): zero
            if constexpr (W == 1) {
                const int S = red_div(32, red_h(d0.m)), lv = red_f32(d0.m) ? 2 : 3;
                auto at     = [&](int t) {
                    const int jj = red_div(t, S), sl = t - jj * S;
                    return cf + ((((jj >> lv) * S + sl) << lv) | (jj & ((1 << lv) - 1)));
                };
#pragma unroll
                for (int r = 0; r < 2; r++)
                    if (lane + 32 * r < end)
                        copy_or_zero(at(lane + 32 * r), A + (r ? d0.ix1 : d0.ix0), lane + 32 * r < ncol);
                for (int t = 64 + lane; t < end; t += 32)
                    *at(t) = 0.f;
            } else {
                using V = std::conditional_t<W % 4 == 0, float4, float2>;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int t = lane + 32 * r;
                    if (t < ncol)
                        copy_row<W>(cf + W * t, A + (long long)W * (r ? d0.ix1 : d0.ix0));
                    else if (t < end)
#pragma unroll
                        for (int i = 0; i < 4 * W / (int)sizeof(V); i++)
                            reinterpret_cast<V *>(cf + W * t)[i] = V{};
                }
            }
            issued++;
            d0 = d1;
            d1 = next_chunk();
        }
        copies_commit();
    };
    DF2 acc[Q]; // W = 1: the low half
#pragma unroll
    for (int s = 0; s < kRedStages - 1; s++)
        issue();
    bool ok  = true;
    int done = 0;
    while (done < issued) {
        const int s = done % kRedStages;
        issue();
        copies_wait<kRedStages - 1>();
        if (!warp_wait_phase(&bar[s], (done / kRedStages) & 1)) {
            ok = false;
            break;
        }
        __syncwarp();
        const unsigned char *st = wbase + (size_t)s * C::kStage;
        const int2 d            = *reinterpret_cast<const int2 *>(st + C::kDesc);
        const int h = red_h(d.x), flags = red_flags(d.x), ncol = red_ncol(d.x);
        const bool f32 = red_f32(d.x);
        const int S = red_div(32, h), slice = red_div(lane, h), row = lane - slice * h, Ln = S * h;
        const float *cf = reinterpret_cast<const float *>(st + C::kCoef);
        const uint4 *D  = reinterpret_cast<const uint4 *>(st) + lane;
        if (flags & kStreamFirst) { // from the dense part where there is one, its loads in flight over the chunk's sums
            const bool add   = (flags & kStreamAdd) && lane < h;
            const float2 *zr = z + d.y + row;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const float2 a = add && 2 * q < nrhs ? zr[(long long)(2 * q) * zlen] : make_float2(0.f, 0.f);
                const float2 b = add && W > 1 && 2 * q + 1 < nrhs ? zr[(long long)(2 * q + 1) * zlen] : make_float2(0.f, 0.f);
                acc[q]         = DF2{fx(a.x, b.x), fx(a.y, b.y)};
            }
        }
        f2x part[Q], part2[Q]; // sums over even and odd columns (W = 1: the halves of part[0])
#pragma unroll
        for (int q = 0; q < Q; q++)
            part[q] = part2[q] = 0ull;
        if (lane < Ln) {
            const int J = red_div(ncol + S - 1, S);
            if constexpr (W == 1) {
                if (f32) {
                    const float4 *cv = reinterpret_cast<const float4 *>(cf) + slice;
#pragma unroll 2
                    for (int g = 0; g < (J + 3) >> 2; g++) {
                        const uint4 w  = D[g * Ln];
                        const float4 c = cv[g * S];
                        part[0]        = fx_fma(fx(__uint_as_float(w.x), __uint_as_float(w.y)), fx(c.x, c.y), part[0]);
                        part[0]        = fx_fma(fx(__uint_as_float(w.z), __uint_as_float(w.w)), fx(c.z, c.w), part[0]);
                    }
                } else {
                    const float4 *cv = reinterpret_cast<const float4 *>(cf) + 2 * slice;
#pragma unroll 2
                    for (int g = 0; g < (J + 7) >> 3; g++) {
                        const uint4 w   = D[g * Ln];
                        const float4 c0 = cv[2 * g * S], c1 = cv[2 * g * S + 1];
                        part[0]         = fx_fma(fx(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u)), fx(c0.x, c0.y), part[0]);
                        part[0]         = fx_fma(fx(__uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u)), fx(c0.z, c0.w), part[0]);
                        part[0]         = fx_fma(fx(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u)), fx(c1.x, c1.y), part[0]);
                        part[0]         = fx_fma(fx(__uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u)), fx(c1.z, c1.w), part[0]);
                    }
                }
            } else {
                // column j of the slice is column slice + S j of the chunk
                auto two = [&](int j, float e0, float e1) {
                    const int t0 = slice + S * j, t1 = t0 + S;
                    f2x x[Q];
                    load_pairs<W>(cf + W * min(t0, kStreamCols - 1), x);
#pragma unroll
                    for (int q = 0; q < Q; q++)
                        part[q] = fx_fma(fx(e0, e0), x[q], part[q]);
                    load_pairs<W>(cf + W * min(t1, kStreamCols - 1), x);
#pragma unroll
                    for (int q = 0; q < Q; q++)
                        part2[q] = fx_fma(fx(e1, e1), x[q], part2[q]);
                };
                if (f32) {
#pragma unroll 1
                    for (int g = 0; g < (J + 3) >> 2; g++) {
                        const uint4 w = D[g * Ln];
                        two(4 * g, __uint_as_float(w.x), __uint_as_float(w.y));
                        two(4 * g + 2, __uint_as_float(w.z), __uint_as_float(w.w));
                    }
                } else {
#pragma unroll 1
                    for (int g = 0; g < (J + 7) >> 3; g++) {
                        const uint4 w = D[g * Ln];
                        two(8 * g, __uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u));
                        two(8 * g + 2, __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
                        two(8 * g + 4, __uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u));
                        two(8 * g + 6, __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
                    }
                }
            }
        }
        if constexpr (W == 1) {
            const float2 p = fx2(part[0]);
            df2_addf(acc[0], fx(p.x + p.y, 0.f));
        } else {
#pragma unroll
            for (int q = 0; q < Q; q++)
                df2_addf(acc[q], fx_add(part[q], part2[q]));
        }
        if (flags & kStreamLast) {
            for (int sl = 1; sl < S; sl++)
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    const int src = (lane + sl * h) & 31;
                    DF2 o;
                    o.s = shfl2(acc[q].s, src);
                    o.c = shfl2(acc[q].c, src);
                    if (slice == 0)
                        acc[q] = df2_add(acc[q], o);
                }
            if (slice == 0) {
                float2 *zr = z + d.y + row;
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    df2_renorm(acc[q]);
                    const bool two = W > 1 && 2 * q + 1 < nrhs, one = 2 * q < nrhs;
                    const float2 vs = fx2(acc[q].s), vc = fx2(acc[q].c);
                    if (one)
                        zr[(long long)(2 * q) * zlen] = make_float2(vs.x, vc.x);
                    if (two)
                        zr[(long long)(2 * q + 1) * zlen] = make_float2(vs.y, vc.y);
                }
            }
        }
        __syncwarp();
        done++;
    }
    copies_wait<0>();
    if (!ok) {
        if (lane == 0)
            atomicExch(status, 2);
        for (int p = done; p < issued; p++)
            if (!warp_wait_phase(&bar[p % kRedStages], (p / kRedStages) & 1) && lane == 0)
                atomicExch(status, 3);
    }
}

// the input of one pass: X for the dense blocks as pair_gather_kernel writes
// it is not enough for the FP32 columns, which take the leading floats of the
// truncating split: [row][w] of them (rows_hi), or [row][w] of its (hi, lo)
// pairs for the phase 1 of one or two right-hand sides
__global__ void red_gather_kernel(const double *__restrict__ x, int ldx, const int *__restrict__ perm, int n, int c0, int w, int mu_src, const int *__restrict__ xexp, int hi_only,
                                  float *__restrict__ out) {
    const long long total = (long long)n * w;
    pdl_next();
    pdl_wait();
    const int shift = 1023 - max(*xexp, 1);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(e / w), c = c0 + (int)(e - (long long)j * w);
        const double v = c < mu_src ? x[(long long)c * ldx + (perm ? perm[j] : j)] : 0.;
        const int ex   = (int)(((unsigned)__double2hiint(v) >> 20) & 0x7FFu);
        F2 f           = (ex == 0 || ex + shift < 1) ? F2{0.f, 0.f} : split64(scale_pow2(v, shift));
        if (ex == 0x7FF)
            f = F2{__int_as_float(0x7fffffff), 0.f};
        if (hi_only)
            out[e] = f.hi;
        else
            reinterpret_cast<float2 *>(out)[e] = make_float2(f.hi, f.lo);
    }
}

// the panels of phase 1 from the reduced tiles: outputs osrc[out ..] (byte
// offsets of their columns), 32 x 32 tiles turned over in shared memory
__global__ void __launch_bounds__(128) red_pack_kernel(const RedPanel *__restrict__ panels, int npanels, const long long *__restrict__ osrc, const unsigned char *__restrict__ mix,
                                                       unsigned char *__restrict__ mirror) {
    __shared__ unsigned tile[4][32][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = gridDim.x * 4;
    for (int p = blockIdx.x * 4 + wid; p < npanels; p += nw) {
        const RedPanel d = panels[p];
        const bool f     = d.kind == kStreamF32;
        const int es = f ? 4 : 2, stride = f ? 16 * ((d.h + 3) >> 2) : 16 * ((d.h + 7) >> 3), hp = stride / es;
        for (int o0 = 0; o0 < hp; o0 += 32) {
            const long long my = o0 + lane < d.h ? osrc[d.out + o0 + lane] : 0;
            for (int k0 = 0; k0 < d.nk; k0 += 32) {
                const int nk = min(32, d.nk - k0);
                __syncwarp();
#pragma unroll 8
                for (int o = 0; o < 32; o++) {
                    const long long so = __shfl_sync(0xffffffffu, my, o);
                    unsigned v         = 0;
                    if (o0 + o < d.h && lane < nk) {
                        const unsigned char *q = mix + so + (long long)es * (k0 + lane);
                        v                      = f ? *reinterpret_cast<const unsigned *>(q) : *reinterpret_cast<const unsigned short *>(q);
                    }
                    tile[wid][lane][o] = v;
                }
                __syncwarp();
                if (o0 + lane < hp)
                    for (int k = 0; k < nk; k++) {
                        unsigned char *q = mirror + d.src + (long long)stride * (k0 + k) + es * (o0 + lane);
                        if (f)
                            *reinterpret_cast<unsigned *>(q) = tile[wid][k][lane];
                        else
                            *reinterpret_cast<unsigned short *>(q) = (unsigned short)tile[wid][k][lane];
                    }
            }
        }
    }
}

int red_sms() {
    int dev = 0, sms = 0;
    HTGPU_CUDA(cudaGetDevice(&dev));
    HTGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max(sms, 1);
}

template <typename K>
void red_smem(K kernel, int bytes, unsigned long long &done) {
    int dev = 0;
    HTGPU_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !(done >> dev & 1)) {
        HTGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        if (dev < 64)
            done |= 1ull << dev;
    }
}

template <int W>
void launch_red1_w(const RedPanel *panels, int npanels, int *ticket, const unsigned char *mirror, const int2 *outs, const float *scale, const float *X, float *A, int *status, cudaStream_t st) {
    static unsigned long long done = 0; // devices whose shared-memory limit was raised
    red_smem(red1_kernel<W>, Red1Cfg<W>::kSmem, done);
    const int nctas = std::min(Red1Cfg<W>::kCtas * red_sms(), (npanels + kRedWarps - 1) / kRedWarps);
    pdl_launch(red1_kernel<W>, nctas, 32 * kRedWarps, Red1Cfg<W>::kSmem, st, panels, npanels, ticket, mirror, outs, scale, X, A, status);
}

template <int W>
void launch_red2_w(const StreamChunk *chunks, const int *rbeg, int nranges, int *ticket, const unsigned char *mix, const int *cidx, const float *A, float2 *z, int zlen, int nrhs, int *status,
                   cudaStream_t st) {
    static unsigned long long done = 0;
    red_smem(red2_kernel<W>, Red2Cfg<W>::kSmem, done);
    const int nctas = std::min(Red2Cfg<W>::kCtas * red_sms(), (nranges + kRedWarps - 1) / kRedWarps);
    pdl_launch(red2_kernel<W>, nctas, 32 * kRedWarps, Red2Cfg<W>::kSmem, st, chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status);
}

} // namespace

void launch_red_gather(const double *x, int ldx, const int *perm, int n, int c0, int w, int mu_src, const int *xexp, bool hi_only, float *out, cudaStream_t st) {
    const long long total = (long long)n * w;
    const int blocks      = (int)std::max<long long>(1, std::min<long long>((total + 255) / 256, 16LL * red_sms()));
    pdl_launch(red_gather_kernel, blocks, 256, 0, st, x, ldx, perm, n, c0, w, mu_src, xexp, hi_only, out);
}

void launch_red_phase1(const RedPanel *panels, int npanels, int *ticket, const unsigned char *mirror, const int2 *outs, const float *scale, const float *X, float *A, int w, int *status, cudaStream_t st) {
    if (npanels <= 0)
        return;
    switch (w) {
    case 1: launch_red1_w<1>(panels, npanels, ticket, mirror, outs, scale, X, A, status, st); break;
    case 2: launch_red1_w<2>(panels, npanels, ticket, mirror, outs, scale, X, A, status, st); break;
    case 4: launch_red1_w<4>(panels, npanels, ticket, mirror, outs, scale, X, A, status, st); break;
    case 6: launch_red1_w<6>(panels, npanels, ticket, mirror, outs, scale, X, A, status, st); break;
    case 8: launch_red1_w<8>(panels, npanels, ticket, mirror, outs, scale, X, A, status, st); break;
    default: require(false, "reduced-precision panels: 1, 2, 4, 6 or 8 right-hand sides a pass"); break;
    }
}

void launch_red_phase2(const StreamChunk *chunks, const int *rbeg, int nranges, int *ticket, const unsigned char *mix, const int *cidx, const float *A, int w, int nrhs, float2 *z, int zlen, int *status,
                       cudaStream_t st) {
    if (nranges <= 0)
        return;
    switch (w) {
    case 1: launch_red2_w<1>(chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status, st); break;
    case 2: launch_red2_w<2>(chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status, st); break;
    case 4: launch_red2_w<4>(chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status, st); break;
    case 6: launch_red2_w<6>(chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status, st); break;
    case 8: launch_red2_w<8>(chunks, rbeg, nranges, ticket, mix, cidx, A, z, zlen, nrhs, status, st); break;
    default: require(false, "reduced-precision chunks: 1, 2, 4, 6 or 8 right-hand sides a pass"); break;
    }
}

void launch_red_pack(const RedPanel *panels, int npanels, const long long *osrc, const unsigned char *mix, unsigned char *mirror, cudaStream_t st) {
    if (npanels <= 0)
        return;
    red_pack_kernel<<<std::min(16 * red_sms(), (npanels + 3) / 4), 128, 0, st>>>(panels, npanels, osrc, mix, mirror);
    HTGPU_CUDA(cudaGetLastError());
}

void set_red_waits(long long cycles) { HTGPU_CUDA(cudaMemcpyToSymbol(g_wait_limit, &cycles, sizeof(cycles))); }

} // namespace htgpu
