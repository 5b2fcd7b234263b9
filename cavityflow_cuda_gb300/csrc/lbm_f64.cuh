// lbm_f64.cuh -- the FP64 collision with its multiplications on the integer
// units.
//
// GB300 has two FP64 lanes an SM: a warp's FP64 instruction takes 16 cycles of
// the SM, in which it could issue 64 others, and the unfused collision (69
// multiplications and 128 additions a cell) is bound by them at 12 % of the
// memory bandwidth.  A product of two doubles needs four 32 x 32 bit multiplies
// and the rounding, about 30 integer instructions, less by a small constant.
// So the multiplications are done there, rounded to nearest even from the
// exact product as IEEE 754 defines it, and run beside the additions, which
// stay on the FP64 units: the same operations in the same order with the same
// results, bit for bit.
//
// The integer products take operands well inside the normal range (exp_ok).
// Zero velocities (the fluid at rest, planes of symmetry) need no product; a
// cell with any other operand outside that range (subnormal, infinite, NaN)
// takes the plain collision.
#pragma once

#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

namespace lbm {
namespace f64 {

__host__ __device__ __forceinline__ uint64_t bits_of(double a)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(a);
#else
    uint64_t u;
    std::memcpy(&u, &a, 8);
    return u;
#endif
}
__host__ __device__ __forceinline__ double from_bits(uint32_t hi, uint32_t lo)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = (uint64_t)hi << 32 | lo;
    double a;
    std::memcpy(&a, &u, 8);
    return a;
#endif
}
__host__ __device__ __forceinline__ uint32_t hi_of(double a) { return (uint32_t)(bits_of(a) >> 32); }
__host__ __device__ __forceinline__ uint32_t lo_of(double a) { return (uint32_t)bits_of(a); }

// |a| in [2^-400, 2^401): products of two such numbers, and those times the
// small constants below, are normal.
__host__ __device__ __forceinline__ bool exp_ok(double a)
{
    return (hi_of(a) & 0x7ff00000u) - ((1023u - 400u) << 20) <= (800u << 20);
}
__host__ __device__ __forceinline__ bool is_zero(double a) { return ((hi_of(a) & 0x7fffffffu) | lo_of(a)) == 0; }

// a * b rounded to nearest even; exponents as exp_ok, or their sum inside the
// normal range.
__host__ __device__ __forceinline__ double mul(double a, double b)
{
    const uint32_t ah = hi_of(a), al = lo_of(a), bh = hi_of(b), bl = lo_of(b);
    const uint32_t am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
    // the product of the 53-bit mantissas, in [2^104, 2^106): hh : (low word of m2) : (low word of ll)
    const uint64_t ll = (uint64_t)al * bl;
    const uint64_t m1 = (uint64_t)am * bl + (ll >> 32);
    const uint64_t m2 = (uint64_t)al * bm + m1;
    const uint64_t hh = (uint64_t)am * bm + (m2 >> 32);
    uint64_t z = hh << 22 | (uint32_t)m2 >> 10;  // its bits 42 .. 105
    const uint32_t rest = (uint32_t)m2 << 22 | (uint32_t)ll;
    const uint32_t sh = (uint32_t)(~z >> 63);     // 1: bit 105 is clear
    z <<= sh;
    uint64_t q = z >> 11;                         // 53 bits, and 11 below them
    const uint32_t below = ((uint32_t)z & 0x7ffu) | (rest != 0 ? 1u : 0u);
    q += below + ((uint32_t)q & 1u) > 0x400u ? 1u : 0u;
    const uint32_t e = (ah & 0x7ff00000u) + (bh & 0x7ff00000u) - (1023u << 20) - (sh << 20);
    return from_bits(((uint32_t)(q >> 32) + e) | ((ah ^ bh) & 0x80000000u), (uint32_t)q);
}

// a * (N / 2^D) for a small odd N whose product with a mantissa needs SH or
// SH + 1 bits more than 53, rounded to nearest even: 3 (SH 1, D 0), 1.5 (1, 1),
// 4.5 (N 9, SH 3, D 1).
template <uint32_t N, uint32_t SH, uint32_t D>
__host__ __device__ __forceinline__ double mul_small(double a)
{
    const uint32_t ah = hi_of(a), al = lo_of(a);
    const uint32_t am = (ah & 0xfffffu) | 0x100000u;
    const uint64_t lo = (uint64_t)al * N;
    const uint64_t v = ((uint64_t)(am * N) << 32) + lo;
    const uint32_t more = (uint32_t)(v >> (53 + SH));  // 0 or 1
    const uint32_t sh = SH + more;
    uint64_t q = v >> sh;
    const uint32_t half = (1u << SH >> 1) << more;
    q = (v + (half - 1u) + ((uint32_t)q & 1u)) >> sh;
    // ah's exponent, sign and the implicit bit of q (q may have become 2^53)
    return from_bits((uint32_t)(q >> 32) + (ah & 0xfff00000u) + ((sh - 1u - D) << 20), (uint32_t)q);
}

__host__ __device__ __forceinline__ double mul3(double a) { return mul_small<3, 1, 0>(a); }
__host__ __device__ __forceinline__ double mul1_5(double a) { return mul_small<3, 1, 1>(a); }
__host__ __device__ __forceinline__ double mul4_5(double a) { return mul_small<9, 3, 1>(a); }

}  // namespace f64
}  // namespace lbm
