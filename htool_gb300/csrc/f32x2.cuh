// Helpers of the warp-fed streaming kernels (pair.cu, red.cu): arithmetic on
// float pairs (.f32x2), double-float accumulators in pairs, and the bounded
// waits and copies of a warp's own ring of shared-memory stages.
#pragma once
#include "df64.cuh"

namespace htgpu {
namespace {

// SM clocks of a wait at most (about 2 s; htgpu_debug_set_waits); one per
// translation unit
__device__ long long g_wait_limit = 4000000000ll;

typedef unsigned long long f2x; // two floats: low word first

__device__ __forceinline__ f2x fx_fma(f2x a, f2x b, f2x c) {
    f2x d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2x fx_add(f2x a, f2x b) {
    f2x d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2x fx_sub(f2x a, f2x b) {
    f2x d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2x fx(float lo, float hi) {
    f2x d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 fx2(f2x v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

struct DF2 { // two double-float accumulators
    f2x s, c;
};

__device__ __forceinline__ void df2_fma(DF2 &a, f2x uh, f2x ul, f2x xh, f2x xl) {
    // two scalar products: the assembler contracts mul.f32x2 and add.f32x2 to
    // one fma in spite of their rounding modifiers, and t = RN(s + uh xh)
    // would lose what TwoSum recovers (the product came out at 9e-9)
    const float2 u = fx2(uh), v = fx2(xh);
    const f2x p  = fx(__fmul_rn(u.x, v.x), __fmul_rn(u.y, v.y));
    const f2x t  = fx_add(a.s, p);
    const f2x nb = fx_sub(a.s, t);              // -(t - s)
    const f2x w  = fx_sub(a.s, fx_add(t, nb)); // what s lost
    f2x l        = fx_fma(uh, xh, nb);          // what the product lost, its own rounding included
    l            = fx_fma(ul, xh, l);
    l            = fx_fma(uh, xl, l);
    a.c          = fx_add(a.c, fx_add(w, l)); // one rounding at c's size, the others at an ulp of s
    a.s          = t;
}

__device__ __forceinline__ void df2_renorm(DF2 &a) {
    const f2x s = fx_add(a.s, a.c);
    a.c         = fx_add(a.c, fx_sub(a.s, s));
    a.s         = s;
}

__device__ __forceinline__ DF2 df2_add(DF2 a, DF2 b) {
    const f2x s  = fx_add(a.s, b.s);
    const f2x nb = fx_sub(a.s, s);
    const f2x w  = fx_sub(a.s, fx_add(s, nb));
    const f2x v  = fx_add(b.s, nb);
    DF2 r;
    r.s = s;
    r.c = fx_add(fx_add(a.c, b.c), fx_add(w, v));
    return r;
}

__device__ __forceinline__ f2x shfl2(f2x v, int src) {
    const float2 f = fx2(v);
    return fx(__shfl_sync(0xffffffffu, f.x, src), __shfl_sync(0xffffffffu, f.y, src));
}

__device__ __forceinline__ unsigned sa(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_try(unsigned long long *b, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(sa(b)), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}

// the whole warp waits for the phase; false when the wait ran out
__device__ __forceinline__ bool warp_wait_phase(unsigned long long *b, unsigned parity) {
    bool ok = mbar_try(b, parity);
    if (!__all_sync(0xffffffffu, ok)) {
        const long long t0 = clock64();
        while (true) {
            ok = mbar_try(b, parity);
            if (__all_sync(0xffffffffu, ok))
                break;
            if (__any_sync(0xffffffffu, clock64() - t0 > g_wait_limit))
                return false;
        }
    }
    return true;
}

// L2 policy for data read once: evicted first, so that the small vectors
// gathered per column stay in L2
__device__ __forceinline__ unsigned long long stream_policy() {
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ void ring_init(unsigned long long *bar, int n) { // lane 0
    for (int s = 0; s < n; s++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&bar[s])) : "memory");
}

// one bulk copy of `bytes` (a multiple of 16, addresses 16-byte aligned)
// completing on the stage's barrier
__device__ __forceinline__ void ring_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar, unsigned long long pol) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(sa(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(sa(dst)), "l"(src), "r"(bytes), "r"(sa(bar)), "l"(pol) : "memory");
}

// Programmatic dependent launch: the kernels of a product follow each other on
// one stream, and each may start (set up its rings, read its descriptors)
// while the one before it ends.  pdl_wait returns when that one has completed
// and its writes are visible; pdl_next lets the next one be launched.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
void pdl_launch(void (*kernel)(P...), int grid, int block, int smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c                             = {};
    c.gridDim                                        = dim3((unsigned)grid);
    c.blockDim                                       = dim3((unsigned)block);
    c.dynamicSmemBytes                               = (size_t)smem;
    c.stream                                         = st;
    c.attrs                                          = at;
    c.numAttrs                                       = 1;
    HTGPU_CUDA(cudaLaunchKernelEx(&c, kernel, P(args)...));
}

template <int B>
__device__ __forceinline__ void copy_async(void *dst, const void *src) {
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(sa(dst)), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

} // namespace
} // namespace htgpu
