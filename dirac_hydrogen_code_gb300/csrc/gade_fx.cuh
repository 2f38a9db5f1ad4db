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
/* two signed limbs of N */
__device__ __forceinline__ int2 fx_split(long long N)
{
    int2 r;
    r.x = (int)((N + (1ll << (FX_LB - 1))) >> FX_LB);
    r.y = (int)(N - ((long long)r.x << FX_LB));
    return r;
}
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }   /* -1022 <= e <= 1023 */
#define FX_NAN 20000                   /* exponents from here on make a sum NaN */
/* acc += V 2^e; e of any size (below the normal range in two factors) */
__device__ __forceinline__ double fx_add(double acc, long long V, int e)
{
    double v = (double)V;
    if (e < -1022) { v *= pow2d(e + 900 < -1022 ? -1022 : e + 900); e = -900; }
    return fma(v, e >= FX_NAN ? __longlong_as_double(0x7FF8000000000000ll) : pow2d(e > 1023 ? 1023 : e), acc);
}
/* the upper 16 bits of a double >= v (v >= 0): sign, exponent and 4 mantissa bits, rounded up */
__device__ __forceinline__ unsigned short fx_bound16(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (unsigned short)((b + 0xFFFFFFFFFFFFull) >> 48);
}
/* the same from the bits of |v|: an infinity or a NaN gives 0x7FF0 */
__device__ __forceinline__ unsigned short fx_bound16_bits(unsigned long long b)
{
    return b >= 0x7FF0000000000000ull ? (unsigned short)0x7FF0 : (unsigned short)((b + 0xFFFFFFFFFFFFull) >> 48);
}
__device__ __forceinline__ double fx_bound_to(unsigned short u) { return __hiloint2double((int)u << 16, 0); }

/*
 * Values with an exponent of their own.  A word (int2, x the low half) holds
 * N in its upper 57 bits (2^55 <= |N| <= 2^56: 53 bits and 3 more) and in its
 * lower 7 an offset, value = N 2^(e - 1078 - offset) with e the exponent of
 * the value's group; zero is N = 0 with offset 127.  A value below 2^-127 of
 * its group's power of two loses bits, any other keeps FP64's.  A factor of
 * the words is X 2^(ex - 1080), |X| <= 2^58 (the larger part of a complex
 * value has ex for its biased exponent).  A sum of up to 15 products aligns
 * its words to its largest product first, C = max (ex - offset); the shifts
 * leave 2^-57 of that product, so the sum is as accurate as FP64's (5 times
 * more, measured on rows with one large product and on rows of equal ones)
 * whichever of its entries is the largest.  Limbs of 30 bits: N / 2^-1 2^-s
 * as h 2^30 + l, l in [0, 2^30), and X as h 2^30 + l, |l| <= 2^29.
 */
#define FX_OFF 127
#define FX_ZERO (-100000)              /* exponent of a zero factor: never the largest */
#define FX_WB 30                       /* bits of the low limb */

__device__ __forceinline__ int2 fx_word_of(long long T, int off)
{
    return make_int2(((int)T & ~FX_OFF) | off, (int)(T >> 32));
}
/* the word of v in a group of exponent e >= v's biased exponent */
__device__ __forceinline__ int2 fx_word(double v, int e)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    int ev = (int)((b >> 52) & 0x7FF);
    long long m = (long long)(b & 0xFFFFFFFFFFFFFull);
    if (ev) m |= 1ll << 52; else ev = 1;
    if (m == 0) return make_int2(FX_OFF, 0);
    int off = e - ev;
    m <<= 10;
    if (off > FX_OFF) { m >>= min(off - FX_OFF, 63); off = FX_OFF; }
    return fx_word_of((long long)b < 0 ? -m : m, off);
}
__device__ __forceinline__ long long fx_shr(long long v, int s)      /* any s >= 0 */
{
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
}
/* 2 N 2^-s as limbs.  The lowest bit is set whatever was shifted out: as
   accurate as rounding to N 2^-s, without a bias and without an addition
   (the offset's bits go the same way) */
__device__ __forceinline__ void fx_take(int wx, int wy, int s, int &h, int &l)
{
    const long long t = fx_shr((long long)(((unsigned long long)(unsigned)wy << 32) | (unsigned)wx), s + 6);
    h = (int)(t >> FX_WB);
    l = ((int)t & ((1 << FX_WB) - 1)) | 1;
}
/* acc += a b.  Written out: from (long long)a * b with a cut from a 64-bit
   value the compiler makes a 64-bit product (12 instructions more for the six
   multiply-adds of a value: 0.49 instead of 0.35 clocks per value and SM) */
__device__ __forceinline__ void fx_mad(long long &acc, int a, int b)
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}
/* limbs of a factor X */
__device__ __forceinline__ int2 fx_limbs(long long X)
{
    int2 r;
    r.x = (int)((X + (1ll << (FX_WB - 1))) >> FX_WB);
    r.y = (int)(X - ((long long)r.x << FX_WB));
    return r;
}
/* the sum of products h 2^60 + m 2^30 (of 2 N and X) in units of 2^58: its
   value is S 2^(e + C - 2101); sums of 30 products stay below 2^62 */
__device__ __forceinline__ long long fx_sum(long long h, long long m)
{
    return (h << 2) + (m >> (FX_WB - 2));
}
/* the same in units of 2^59, to nearest: S 2^(e + C - 2100); sums of 66 products
   stay below 2^63 */
__device__ __forceinline__ long long fx_sum59(long long h, long long m)
{
    return 2 * h + ((m + (1ll << (FX_WB - 2))) >> (FX_WB - 1));
}
/* the value of a word in a group of exponent e */
__device__ __forceinline__ double fx_value(int2 w, int e)
{
    const long long v = (long long)(((unsigned long long)(unsigned)w.y << 32) | (unsigned)(w.x & ~FX_OFF));
    return fx_add(0.0, v >> 7, e - 1078 - (w.x & FX_OFF));
}
/* S 2^max(C, Cb) as the sum of S 2^C and Sb 2^Cb (a shift loses 2^-55 of the
   largest product) */
__device__ __forceinline__ void fx_join(long long &S, int C, long long Sb, int Cb)
{
    S = fx_shr(S, max(Cb - C, 0)) + fx_shr(Sb, max(C - Cb, 0));
}

#endif
