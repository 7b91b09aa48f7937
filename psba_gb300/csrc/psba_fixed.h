// Sums of FP64 products in block fixed point, on the integer pipe.
//
// GB300's FP64 pipe does two multiply-adds per clock and SM; its integer pipe
// does 28 of the 32 x 32 + 64-bit multiply-adds (both measured).  A sum of
// products whose factors are brought to a common exponent and cut into two
// signed 29-bit limbs takes three of those per product, so it runs at more
// than four times the FP64 rate.
//
// Two limbs alone would hold a factor to 57 bits below the largest of its
// block, where FP64 keeps 53 bits of each one's own: less, where the factors of
// a block are more than four binary orders apart.  A factor therefore has a
// third piece, the 16 bits below its limbs, and what the three products of
// limbs leave out (low limb by low limb, third piece by high limb) is summed
// in FP32 beside them: it stands 57 bits below the largest product, so FP32's
// 24 bits bring the sums to about 73 bits below it.  Against 80-bit sums of
// the same factors, relative to the sum of the products' magnitudes (rms, in
// units of 2^-53; FP64 multiply-adds in brackets): 0.3-0.5 (0.4-0.8) on scenes of
// 7 to 21 cameras, 0.15 (0.22) with depths over a factor of 2,000, 0.72 (1.6)
// with standard deviations from 1e-6 to 1e6 besides; 0.6-1.3, 4 and 1,270 with the limbs alone.
#pragma once

#include <cuda_runtime.h>

namespace psba {

// One observation's rows: their limbs as int2 words, [j][row] with the rows padded
// to a multiple of a thread's tile (6 -> 6, 11 -> 12, 16 -> 16 rows), then
// their third pieces, 16 bits each, [j][group][4] with fx_group rows a group
__host__ __device__ constexpr int fx_rows(int cnp) { return cnp == 11 ? 12 : cnp; }
__host__ __device__ constexpr int fx_group(int cnp) { return cnp == 16 ? 4 : 3; }
__host__ __device__ constexpr int fx_limb_words(int cnp) { return 3 * fx_rows(cnp); }
__host__ __device__ constexpr int fx_low_words(int cnp) { return 3 * fx_rows(cnp) / fx_group(cnp); }
__host__ __device__ constexpr int fx_words(int cnp) { return fx_limb_words(cnp) + fx_low_words(cnp); }

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

// A factor with its third piece: hi 2^29 + lo + f 2^-16, 0 <= f < 2^16
struct Fx3 {
    int2 v;
    unsigned f;
};

// (v + f 2^-16) 2^-d, d >= 0, cut below
__device__ __forceinline__ Fx3 fx_cut(long long v, unsigned f, int d)
{
    const unsigned low = d < 16 ? ((unsigned)v << 16 | f) >> d : (unsigned)(v >> min(d - 16, 63));
    return Fx3{fx_split(v >> min(d, 63)), low & 0xffffu};
}

// x in units of 2^(E - 1023 - 56), d = E - fx_exp(x) >= 0
__device__ __forceinline__ Fx3 fx_limbs3(double x, int d)
{
    const int h = __double2hiint(x);
    const unsigned m1 = (unsigned)(h & 0xfffff) | ((h & 0x7ff00000) ? 0x100000u : 0u);
    const long long m = (long long)((unsigned long long)m1 << 32 | (unsigned)__double2loint(x)) << 4;
    return fx_cut(h < 0 ? -m : m, 0, d);
}

// moved d >= 0 bits down
__device__ __forceinline__ Fx3 fx_shift(int2 a, unsigned f, int d)
{
    return fx_cut(((long long)a.y << FX_LIMB) + a.x, f, d);
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

// A tile's factors as FP32, for what the limbs' products leave out
template <int N>
struct FxLow {
    float hi[N], lo[N], f[N];
};

// scale: 2^-13 on one of the two sides, so that lo lo' has the unit of hi f' (2^13 limb units)
template <int N>
__device__ __forceinline__ void fx_low(const int2 (&v)[N], const float (&f)[N], float scale, FxLow<N> &o)
{
#pragma unroll
    for (int k = 0; k < N; ++k) {
        o.hi[k] = (float)v[k].y;
        o.lo[k] = (float)v[k].x * scale;
        o.f[k] = f[k];
    }
}

// a b^T into the sums of hi hi, of the cross terms and of the rest
template <int TR, int TC>
__device__ __forceinline__ void fx_products(const int2 (&a)[TR], const float (&fa)[TR], const int2 (&b)[TC],
                                            const float (&fb)[TC], long long (&hh)[TR][TC], long long (&hl)[TR][TC],
                                            float (&cr)[TR][TC])
{
    FxLow<TR> u;
    FxLow<TC> w;
    fx_low(a, fa, 0x1p-13f, u);
    fx_low(b, fb, 1.0f, w);
#pragma unroll
    for (int p = 0; p < TR; ++p)
#pragma unroll
        for (int q = 0; q < TC; ++q) {
            fx_mad(a[p], b[q], hh[p][q], hl[p][q]);
            cr[p][q] = fmaf(u.lo[p], w.lo[q], fmaf(u.hi[p], w.f[q], fmaf(u.f[p], w.hi[q], cr[p][q])));
        }
}

// The sum hh 2^58 + hl 2^29 + cr 2^13 (12 products at most) as H 2^58 + L 2^29,
// 0 <= L < 2^29: the L of eight such sums add up below 2^32.
__device__ __forceinline__ void fx_carry(long long hh, long long hl, float cr, long long &H, unsigned &L)
{
    fx_madw(hl, __float2int_rn(cr * 0x1p-20f), 16);  // |cr| < 2^49
    H = hh + (hl >> FX_LIMB);
    L = (unsigned)hl & ((1u << FX_LIMB) - 1);
}

// acc + (H + L 2^-29) 2^(e - FX_BIAS): as many of L's bits behind H's as 64 hold
__device__ __forceinline__ double fx_add(double acc, long long H, unsigned L, int e)
{
    H += L >> FX_LIMB;
    L &= (1u << FX_LIMB) - 1;
    const int s = min(FX_LIMB, __clzll(H ^ (H >> 63)) - 1);
    return fx_add(acc, (long long)((unsigned long long)H << s) | (L >> (FX_LIMB - s)), e - s);
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
