// Sums of FP64 products in block fixed point, on the integer pipe.
//
// GB300's FP64 pipe does two multiply-adds per clock and SM; its integer pipe
// does 28 of the 32 x 32 + 64-bit multiply-adds (both measured).  A sum of
// products whose factors are brought to a common exponent and cut into two
// signed 29-bit limbs takes three of those per product, so it runs at more
// than four times the FP64 rate.  Its accuracy: a factor is cut 57 bits below the
// largest of its block (FP64 keeps 53 bits of its own), the product of the two
// low limbs (2^-58 of the largest product) is left out, and the sums
// themselves are exact, where an FP64 sum rounds every addition to 53 bits.
#pragma once

#include <cuda_runtime.h>

namespace psba {

// int2 words of one observation's rows in limbs, [j][row] with the rows padded
// to a multiple of a thread's tile: 6 -> 6, 11 -> 12, 16 -> 16 rows
__host__ __device__ constexpr int fx_rows(int cnp) { return cnp == 11 ? 12 : cnp; }
__host__ __device__ constexpr int fx_words(int cnp) { return 3 * fx_rows(cnp); }

#ifdef __CUDACC__
constexpr int FX_LIMB = 29;          // bits of the low limb (signed, centred)
constexpr int FX_NAN = 1 << 24;      // exponent of rows with an infinity or a NaN
// a sum's value is T 2^(E - FX_BIAS) for limbs aligned to exponent fields that
// add up to E: two biases of 1023, twice 56 fraction bits, less the 58 that
// T = sum hi hi + (sum of cross terms) 2^-29 stands above
constexpr int FX_BIAS = 2 * 1023 + 2 * 56 - 2 * FX_LIMB;

// The exponent field of x; zeros and subnormals count as the smallest
// exponent (their fraction has no implicit one).
__device__ __forceinline__ int fx_exp(double x) { return max((__double2hiint(x) >> 20) & 0x7ff, 1); }
__device__ __forceinline__ bool fx_nonfinite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

// v as v = hi 2^29 + lo, -2^28 <= lo < 2^28; .x = lo, .y = hi
__device__ __forceinline__ int2 fx_split(long long v)
{
    v += 1LL << (FX_LIMB - 1);
    return make_int2((int)((unsigned)v & ((1u << FX_LIMB) - 1)) - (1 << (FX_LIMB - 1)), (int)(v >> FX_LIMB));
}

// x in units of 2^(E - 1023 - 56), d = E - fx_exp(x) >= 0 (|hi| <= 2^28)
__device__ __forceinline__ int2 fx_limbs(double x, int d)
{
    const int h = __double2hiint(x);
    const unsigned m1 = (unsigned)(h & 0xfffff) | ((h & 0x7ff00000) ? 0x100000u : 0u);
    unsigned long long m = ((unsigned long long)m1 << 32 | (unsigned)__double2loint(x)) << 4;
    m >>= min(d, 63);
    return fx_split(h < 0 ? -(long long)m : (long long)m);
}

// limbs moved d >= 0 bits down
__device__ __forceinline__ int2 fx_shift(int2 a, int d)
{
    return fx_split((((long long)a.y << FX_LIMB) + a.x) >> min(d, 63));
}

// c += a b.  Written as a wide product and an addition, which the assembler
// fuses into one instruction; given mad.wide.s32 (or the C expression) it
// issues the two apart when the operands come from memory (counted; 27.7
// against 24 multiply-adds per clock and SM).
__device__ __forceinline__ void fx_madw(long long &c, int a, int b)
{
    asm("{ .reg .s64 t; mul.wide.s32 t, %1, %2; add.s64 %0, %0, t; }" : "+l"(c) : "r"(a), "r"(b));
}

// One product into the sums of hi hi and of the cross terms.
__device__ __forceinline__ void fx_mad(int2 a, int2 b, long long &hh, long long &hl)
{
    fx_madw(hh, a.y, b.y);
    fx_madw(hl, a.y, b.x);
    fx_madw(hl, a.x, b.y);
}

__device__ __forceinline__ long long fx_total(long long hh, long long hl)
{
    return hh + ((hl + (1LL << (FX_LIMB - 1))) >> FX_LIMB);
}

// acc + T 2^(e - FX_BIAS)
__device__ __forceinline__ double fx_add(double acc, long long T, int e)
{
    const int b = e - FX_BIAS + 1023;
    if (b >= 1 && b <= 2046) return fma((double)T, __hiloint2double(b << 20, 0), acc);
    return acc + ldexp((double)T, e - FX_BIAS);
}

// The weight of a camera's row r: its size, as the exponent of sqrt(U_rr)
// (U = sum A^T A), so that rows of different units (radians, metres, pixels)
// share an observation's exponent.  Any value is right; a closer one loses
// fewer bits.
__device__ __forceinline__ int fx_weight(double u_rr) { return (fx_exp(u_rr) - 1023) >> 1; }

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}
#endif

}  // namespace psba
