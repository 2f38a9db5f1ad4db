/*
 * gade_fx.cuh - fixed-point products of FP64 values on the integer units
 * (device helpers shared by the operator and the projection kernels).
 */
#ifndef GADE_FX_CUH
#define GADE_FX_CUH

/*
 * GB300 retires 2 DFMA per clock and SM but 32 32x32+64-bit integer
 * multiply-adds (measured: 1.6 against 24 per nominal clock), so the long
 * real x real sums of the assembled operator run there.  A vector of FP64
 * values that share a power of two is held as integers N, value = N 2^e:
 *   matrix values     |N| <= 2^57, one e per row or run        (FX_UPA = 4)
 *   vector entries    |N| <= 2^58, one e per staged window     (FX_UPX = 5)
 * each in two signed limbs, N = hi 2^29 + lo, |lo| <= 2^28.  A product is
 * hi hi 2^58 + (hi lo + lo hi) 2^29, three multiply-adds into two 64-bit
 * sums (the lo lo term, below 2^-56 of the largest product, is left out);
 * sums of up to 32 products stay below 2^63 and are exact.  A 53-bit
 * mantissa is held in full down to 2^-4 (2^-5 for vector entries) of its
 * group's largest value and rounded to nearest below that, at 2^-58 (2^-59)
 * of the group's power of two, so a row's sum carries an error of about 2^-57
 * of its largest terms once, where FP64 rounds every product and partial sum
 * to 2^-53 of them.
 */
#define FX_UPA 4
#define FX_UPX 5
#define FX_LB 29                       /* bits of the low limb */

/* biased exponent field of a double given by its high word */
__host__ __device__ __forceinline__ int fx_exp(unsigned hi) { return (int)((hi >> 20) & 0x7FF); }

/* a mantissa already shifted up, down by the exponent difference d >= 0, to nearest */
__device__ __forceinline__ unsigned long long fx_shift(unsigned long long m, int d)
{
    return d ? ((m >> (d > 64 ? 63 : d - 1)) + 1) >> 1 : m;
}
/* N of v in a group whose largest biased exponent is em (finite, em >= the
   value's own): the mantissa shifted up by `up` bits and down by the
   exponent difference; v = N 2^(em - 1075 - up) */
__device__ __forceinline__ long long fx_from(double v, int em, int up)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    int ev = (int)((b >> 52) & 0x7FF);
    unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    if (ev) m |= 1ull << 52; else ev = 1;
    m = fx_shift(m << up, em - ev);
    return (long long)b < 0 ? -(long long)m : (long long)m;
}
/* the same for a float, |N| <= 2^57, in a group whose largest biased float
   exponent is em: v = N 2^(em - 183) */
__device__ __forceinline__ long long fx_from_float(float v, int em)
{
    const unsigned b = __float_as_uint(v);
    int ev = (int)((b >> 23) & 0xFF);
    unsigned long long m = b & 0x7FFFFFu;
    if (ev) m |= 1ull << 23; else ev = 1;
    m = fx_shift(m << 33, em - ev);
    return (int)b < 0 ? -(long long)m : (long long)m;
}
/* two signed limbs of N */
__device__ __forceinline__ int2 fx_split(long long N)
{
    int2 r;
    r.x = (int)((N + (1ll << (FX_LB - 1))) >> FX_LB);
    r.y = (int)(N - ((long long)r.x << FX_LB));
    return r;
}
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }   /* -1022 <= e <= 1023 */
/* acc += V 2^e; e of any size (below the normal range in two factors) */
__device__ __forceinline__ double fx_add(double acc, long long V, int e)
{
    double v = (double)V;
    if (e < -1022) { v *= pow2d(e + 900 < -1022 ? -1022 : e + 900); e = -900; }
    return fma(v, pow2d(e > 1023 ? 1023 : e), acc);
}
/* the upper 16 bits of a double >= v (v >= 0): sign, exponent and 4 mantissa bits, rounded up */
__device__ __forceinline__ unsigned short fx_bound16(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (unsigned short)((b + 0xFFFFFFFFFFFFull) >> 48);
}
__device__ __forceinline__ double fx_bound_to(unsigned short u) { return __hiloint2double((int)u << 16, 0); }

#endif
