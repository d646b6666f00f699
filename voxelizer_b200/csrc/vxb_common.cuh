// Helpers shared by the kernel files.
#pragma once

#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace vxb {
namespace detail {

struct D3 { double x, y, z; };
struct F3 { float x, y, z; };

__device__ __forceinline__ uint32_t laneMaskLt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Unit of element x: the largest u < n with base[u] <= x (base[0] = 0).
template <class T>
__device__ __forceinline__ uint32_t unitOf(const T* __restrict__ base, uint32_t n, T x) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Largest t < n with off[t] <= item (off[n] > item), by a 32-way search of
// the whole warp: ceil(log32 n) dependent loads.
__device__ __forceinline__ uint32_t warpFindOwner(const uint32_t* __restrict__ off, uint32_t n, uint32_t item,
                                                  uint32_t lane) {
    uint32_t lo = 0, hi = n;  // off[lo] <= item < off[hi]
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31u) / 32u;
        const uint32_t p = lo + lane * step;
        const bool ok = p < hi && __ldg(off + p) <= item;
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        const uint32_t nlo = lo + (31u - (uint32_t)__clz(m)) * step;
        hi = min(nlo + step, hi);
        lo = nlo;
    }
    return lo;
}

// Exact conversion of a 32-bit unsigned integer: 2^52 + x as a bit pattern,
// less 2^52 (the conversion instruction runs at a quarter of the FP64 rate).
__device__ __forceinline__ double toDouble(uint32_t x) {
    return __dsub_rn(__hiloint2double(0x43300000, (int)x), 4503599627370496.0);
}

// Whether |x| lies in [2^-400, 2^400) (not zero, infinite or NaN).
__host__ __device__ __forceinline__ bool divScale(double x) {
#ifdef __CUDA_ARCH__
    const uint32_t h = (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    const uint32_t h = (uint32_t)(u >> 32);
#endif
    return (h & 0x7FFFFFFFu) - 0x26F00000u < 0x32000000u;
}

// The correctly rounded x / d for operands with divExact(x) and r = 1 / d
// rounded to nearest with divScale(d).  Two corrections of x * r by its
// remainder: the first brings the quotient within one ulp, and the second
// then rounds it correctly (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990, theorem 7).  With both operands within 2^+-400 no intermediate
// leaves the normal range; x = +-0 gives a zero (of either sign).
__device__ __forceinline__ bool divExact(double x) { return divScale(x) || x == 0.0; }
__device__ __forceinline__ double divBy(double x, double d, double r) {
    double q = __dmul_rn(x, r);
    q = __fma_rn(__fma_rn(-q, d, x), r, q);
    return __fma_rn(__fma_rn(-q, d, x), r, q);
}

// The same in FP32, for operands within 2^+-60.
__host__ __device__ __forceinline__ bool divScaleF(float x) {
#ifdef __CUDA_ARCH__
    const uint32_t h = __float_as_uint(x);
#else
    uint32_t h;
    memcpy(&h, &x, 4);
#endif
    return (h & 0x7FFFFFFFu) - 0x21800000u < 0x3C000000u;
}
__device__ __forceinline__ bool divExactF(float x) { return divScaleF(x) || x == 0.0f; }
__device__ __forceinline__ float divByF(float x, float d, float r) {
    float q = __fmul_rn(x, r);
    q = __fmaf_rn(__fmaf_rn(-q, d, x), r, q);
    return __fmaf_rn(__fmaf_rn(-q, d, x), r, q);
}

// Blocks for `work` items at `threads` per block, capped (grid-stride loops).
inline uint32_t gridFor(uint64_t work, uint32_t threads, uint32_t cap = 148u * 32u) {
    uint64_t b = (work + threads - 1) / threads;
    if (b == 0) b = 1;
    return (uint32_t)(b < cap ? b : cap);
}

// 1 / d for divBy and divByF.
inline double divReciprocal(double d) { return divScale(d) ? 1.0 / d : 0.0; }
inline float divReciprocalF(float d) { return divScaleF(d) ? 1.0f / d : 0.0f; }

}  // namespace detail
}  // namespace vxb
