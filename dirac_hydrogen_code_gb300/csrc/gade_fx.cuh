/*
 * gade_fx.cuh - sums of products of FP64 values on the integer units (device
 * helpers shared by the operator, the block solves and the projection).
 */
#ifndef GADE_FX_CUH
#define GADE_FX_CUH

/*
 * GB300 retires 2 DFMA per clock and SM but some 27 32x32+64-bit integer
 * multiply-adds (measured: 1.6 against 24-27 per nominal clock), so long sums
 * of products run there.
 *
 * A matrix value is a word (int2, x the low half): N in its upper 57 bits
 * (2^55 <= |N| <= 2^56: 53 bits and 3 more) and an offset in its lower 7,
 * value = N 2^(e - 1078 - offset) with e the exponent of the value's group;
 * zero is N = 0 with offset 127.  A value below 2^-127 of its group's power of
 * two loses bits, any other keeps FP64's.  (Factors and basis entries use the
 * 7 bits for an exponent of their own.)  A vector entry is X 2^(ex - 1080),
 * |X| <= 2^58, with ex the biased exponent of the larger part of the complex
 * entry.
 *
 * A sum of up to 33 complex or 30 real products aligns its words to its
 * largest product first, C = max (ex - offset): each N is shifted into place
 * and multiplied in limbs of 30 bits, 2 N 2^-s = h 2^30 + l with l in
 * [0, 2^30) and X = h 2^30 + l with |l| <= 2^29, three multiply-adds per
 * product into two 64-bit sums (l l is left out: below 2^-54 of the largest
 * product).  The shifts leave 2^-57 of that product, so a sum's error is a few
 * 2^-54 of its largest product, whichever of its entries is the largest;
 * FP64 rounds every product and partial sum to 2^-53 of its own.  (With one
 * exponent per row of values and per window of entries the shift and the
 * offsets are not needed, and a row whose own products are far below the
 * largest value times the largest entry loses its digits.)
 */
#define FX_UPX 5                       /* bits of X below a 53-bit value */
#define FX_OFF 127
#define FX_ZERO (-100000)              /* exponent of a zero factor: never the largest */
#define FX_WB 30                       /* bits of the low limb */

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
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }   /* -1022 <= e <= 1023 */
#define FX_NAN 20000                   /* exponents from here on make a sum NaN */
/* acc += V 2^e; e of any size (below the normal range in two factors) */
__device__ __forceinline__ double fx_add(double acc, long long V, int e)
{
    double v = (double)V;
    if (e < -1022) { v *= pow2d(e + 900 < -1022 ? -1022 : e + 900); e = -900; }
    return fma(v, e >= FX_NAN ? __longlong_as_double(0x7FF8000000000000ll) : pow2d(e > 1023 ? 1023 : e), acc);
}
/* the upper 16 bits of a double >= |v|, given the bits of |v|: exponent and 4
   mantissa bits, rounded up; an infinity or a NaN gives 0x7FF0 */
__device__ __forceinline__ unsigned short fx_bound16_bits(unsigned long long b)
{
    return b >= 0x7FF0000000000000ull ? (unsigned short)0x7FF0 : (unsigned short)((b + 0xFFFFFFFFFFFFull) >> 48);
}
__device__ __forceinline__ double fx_bound_to(unsigned short u) { return __hiloint2double((int)u << 16, 0); }

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
