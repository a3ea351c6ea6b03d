// Small arithmetic of the kernels that tests compile for the host, without a GPU.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define UG_HD __host__ __device__ __forceinline__
#define UG_HD_CALL static __host__ __device__ __noinline__
#else
#define UG_HD inline
#define UG_HD_CALL inline
#endif

namespace ug {

// Where a list of noise events (cap entries, the last one kept for its mark) goes on: at its
// start, or, resumed, behind the mark at `at` that its last segment ended with.  A full list has
// that mark in its last entry; it goes on there, where only the next mark is written, over it.
UG_HD int list_start(bool resume, int at, int cap)
{
    return !resume ? 0 : at + 1 < cap ? at + 1 : cap - 1;
}

UG_HD uint32_t double_hi(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    return (uint32_t)(b >> 32);
#endif
}
UG_HD uint32_t double_lo(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    return (uint32_t)b;
#endif
}

UG_HD_CALL double div_rare(double x, double d) { return x / d; }

// x / d correctly rounded, z = RN(1/d), for a d > 0 whose odd part D is below 2^50 (Markstein's
// division by a known divisor: one correction of x z by its remainder).  q is within 1.5 ulp of
// x / d, its remainder r is exact (a multiple of D's unit below 1.5 D), and q + r z is off by at
// most 1.5 2^-53 ulp before the last rounding, while x / d is at least 1 / (2 D) ulp away from
// the middle of two doubles.  Quotients near the ends of the range, infinities and NaN take the
// division; zeros keep their sign.
UG_HD double div_known(double x, double d, double z)
{
    const double q = x * z;
    double a = fma(fma(-d, q, x), z, q);
    const uint32_t e = (double_hi(q) >> 20) & 0x7ffu;
    if (e - 0x80u >= 0x770u) {
        const bool zero = ((double_hi(x) << 1) | double_lo(x)) == 0;
        a = zero ? x : div_rare(x, d);
    }
    return a;
}

}  // namespace ug
