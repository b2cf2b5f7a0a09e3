// Shared host/device helpers of libashb200 (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "ashb200.h"

namespace ashb {

// ---- host-side error plumbing -------------------------------------------------
void set_error(const char* fmt, ...);

#define ASHB_CUDA_TRY(expr)                                                              \
    do {                                                                                 \
        cudaError_t _e = (expr);                                                         \
        if (_e != cudaSuccess) {                                                         \
            ::ashb::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),    \
                              __FILE__, __LINE__);                                       \
            return ASHB_ERR_CUDA;                                                        \
        }                                                                                \
    } while (0)

#define ASHB_REQUIRE(cond, ...)               \
    do {                                      \
        if (!(cond)) {                        \
            ::ashb::set_error(__VA_ARGS__);   \
            return ASHB_ERR_INVALID;          \
        }                                     \
    } while (0)

// Launch check: catches configuration errors without synchronising.
#define ASHB_LAUNCH_CHECK() ASHB_CUDA_TRY(cudaGetLastError())

// Number of SMs of the current device (148 on B200); cached per process.
int sm_count();

// Grid size for a grid-stride kernel: a whole number of waves of resident CTAs.
inline unsigned wave_grid(int64_t work_items, int threads, int ctas_per_sm) {
    int64_t need = (work_items + threads - 1) / threads;
    int64_t wave = (int64_t)sm_count() * ctas_per_sm;
    if (need < 1) need = 1;
    if (need <= wave) return (unsigned)need;
    int64_t waves = (need + wave - 1) / wave;
    if (waves > 8) waves = 8;
    return (unsigned)(waves * wave);
}

// ---- device helpers -----------------------------------------------------------
__device__ __forceinline__ uint32_t fmix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return h;
}

// Slot hash of a packed int32 key (unused columns are zero).  A column is folded in by a multiplication whose high bits are
// brought down before the next (xorshift-multiply; the odd multipliers of 32-bit hash-prospector searches): 14
// operations for three columns.  With a full murmur3 finaliser per column it was 27, half of a ray march's probe (a view
// of 307,200 rays 236 us, 214 now).  Chains are as long as random slots' for lattices of strides up to 2^18 in each
// column, alike or mixed, for planes, lines, diagonals, clusters and the bits of floats; where only the uppermost bits of
// columns differ (strides of 2^22 and more, mixed) they are up to a third longer on average.  Those of a plain linear
// combination of the columns are more than twice as long at strides of 2^16.
__device__ __forceinline__ uint32_t hash_key(int k0, int k1, int k2, int k3) {
    uint32_t h = (uint32_t)k0 * 0x9E3779B1u;
    h ^= h >> 15;
    h = h * 0x2C1B3C6Du + (uint32_t)k1 * 0x85EBCA77u;
    h ^= h >> 15;
    h = h * 0x297A2D39u + (uint32_t)k2 * 0xC2B2AE3Du;
    if (k3 != 0) {
        h ^= h >> 15;
        h = h * 0x846CA68Bu + (uint32_t)k3 * 0x27D4EB2Fu;
    }
    h ^= h >> 16;
    h *= 0x7FEB352Du;
    return h ^ (h >> 15);
}

// Twice the bits of the smallest of four magnitudes, less one: zeros wrap and count as the largest.
__device__ __forceinline__ uint32_t least_magnitude(float a, float b, float c, float e) {
    return min(min(2u * __float_as_uint(a) - 1u, 2u * __float_as_uint(b) - 1u),
               min(2u * __float_as_uint(c) - 1u, 2u * __float_as_uint(e) - 1u));
}
__device__ __forceinline__ bool all_zero(float a, float b, float c, float e) { return least_magnitude(a, b, c, e) == 0xFFFFFFFFu; }

// Quotients that share a positive divisor, each equal to __fdiv_rn(a, d) bit for bit.  Markstein's theorem (P. Markstein,
// IBM J. Res. Dev. 34, 1990): with y = RN(1 / d) and q within one unit of a / d, q - (q d - a) y rounds to RN(a / d).
// a * y is within two units, one correction brings it within one and the second is the theorem's: one reciprocal and five
// operations a quotient.  Holds where nothing over- or underflows, and for zeros (which keep their sign); `exact` says
// whether it does for a numerator, the caller divides where not.
struct SharedDivisor {
    float d, y;
    bool plain;
    __device__ __forceinline__ explicit SharedDivisor(float divisor) {
        d = divisor;
        y = __frcp_rn(divisor);
        plain = divisor >= 0x1p-30f && divisor <= 0x1p30f;
    }
    __device__ __forceinline__ bool exact(float a, float b, float c, float e) const {
        const float most = fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fabsf(e)));   // a NaN divides to NaN either way
        return plain && most <= 0x1p90f && least_magnitude(a, b, c, e) >= 2u * 0x12800000u - 1u;   // 2^-90
    }
    __device__ __forceinline__ float quotient(float a) const {
        float q = __fmul_rn(a, y);
        q = __fmaf_rn(-__fmaf_rn(q, d, -a), y, q);
        return __fmaf_rn(-__fmaf_rn(q, d, -a), y, q);
    }
    // The N numerators of `a` divided in place.
    template <int N>
    __device__ __forceinline__ void divide(float (&a)[N]) const {
        static_assert(N >= 1 && N <= 4, "");
        if (exact(a[0], a[N > 1], a[N > 2 ? 2 : 0], a[N - 1])) {
#pragma unroll
            for (int k = 0; k < N; ++k) a[k] = quotient(a[k]);
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                asm volatile("" : "+f"(a[k]));   // or both sides are computed and one is picked
                a[k] = __fdiv_rn(a[k], d);
            }
        }
    }
};

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

}  // namespace ashb
