// FP64 numbers to and from 64-bit fixed point, and fixed-point products, for the integer pipes: the
// FP64 pipe of sm_103a takes a warp instruction every 64 cycles and SM partition.
#pragma once

#include <cuda_runtime.h>

namespace cg {

// exponent of a row with an infinity or a NaN: what it enters becomes NaN
constexpr int kNonFinite = 1 << 20;

// u 2^s in FP64 (one rounding; flushed to zero below the normal range)
__device__ __forceinline__ double scaled(long long u, int s)
{
    const double x = __ll2double_rn(u);
    const int hi = __double2hiint(x), e = ((hi >> 20) & 0x7ff) + s;
    if (s > kNonFinite / 2) return __longlong_as_double(0x7ff8000000000000ll);
    if (u == 0 || e <= 0) return 0.0;
    if (e >= 0x7ff) return __hiloint2double((hi & 0x80000000) | 0x7ff00000, 0);
    return __hiloint2double(hi + (s << 20), __double2loint(x));
}

__device__ __forceinline__ int exp_field(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// v as 2^(e - FB) X, |v| < 2^e, X rounded to the nearest; FB <= 62
template <int FB = 54>
__device__ __forceinline__ long long to_fixed(double v, int e)
{
    const long long bits = __double_as_longlong(v);
    const int f = (int)((unsigned long long)bits >> 52) & 0x7ff;
    const unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
    int r = e - (f - 1022);
    if (f == 0 || r > FB + 1) return 0;
    if (r < 0) r = 0;  // only with a non-finite entry, whose row is marked
    const long long x = (long long)(((m << (FB - 52) >> r) + 1) >> 1);
    return bits < 0 ? -x : x;
}

// u 2^s in FP64, rounded to the nearest, the signs flipped by `flip` (0 or 0x80000000): __ll2double_rn is one
// FP64-pipe instruction more per number, and that pipe is the scarcest (with one, two, three of four numbers
// through it the update of a factorisation took 1, 4, 10 % longer).  Numbers below 2^32 and results that may
// not be normal take one branch for all N, so that the N chains of the usual case interleave.
template <int N>
__device__ __forceinline__ void scaled_ints(const long long (&u)[N], const int (&s)[N], unsigned flip, double (&x)[N])
{
    unsigned low = 0xffffffffu;
    int smin = s[0], smax = s[0];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int hi = (int)(u[i] >> 32), sg = hi >> 31;
        const unsigned long long a = (unsigned long long)((u[i] ^ sg) - sg);
        const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
        const int lz = __clz((int)ah);
        low = min(low, ah);
        smin = min(smin, s[i]);
        smax = max(smax, s[i]);
        const unsigned nh = __funnelshift_l(al, ah, lz), nl = al << (lz & 31);
        const unsigned long long m = (((unsigned long long)(nh >> 11) << 32) | __funnelshift_r(nl, nh, 11)) +
                                     ((nl >> 10) & 1u) +  // 1085 - lz + s: the exponent field less one
                                     ((unsigned long long)((unsigned)(1085 + s[i] - lz) << 20) << 32);
        x[i] = __hiloint2double((int)((unsigned)(m >> 32) | (((unsigned)sg ^ flip) & 0x80000000u)), (int)(unsigned)m);
    }
    if (low == 0 || smin < -1021 || smax > 959) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const double y = scaled(u[i], s[i]);
            x[i] = __hiloint2double(__double2hiint(y) ^ (int)flip, __double2loint(y));
        }
    }
}
__device__ __forceinline__ double scaled_int(long long u, int s, unsigned flip)
{
    const long long v[1] = {u};
    const int t[1] = {s};
    double x[1];
    scaled_ints<1>(v, t, flip, x);
    return x[0];
}

// ---- FP64 multiplication in integers, to the bit ----------------------------------------------

// the 53-bit significand of a normal number, its top bit at bit 63
__device__ __forceinline__ unsigned long long significand(double v)
{
    return (((unsigned long long)__double_as_longlong(v) & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
}

// The product of two significands, rounded to the nearest (even) as an FP64 multiplication rounds: `shift`
// counts the products below 2, and the top bit of `valid` goes where rounding carried past the top (such a
// product is left to the caller).
__device__ __forceinline__ unsigned long long mul_significand(unsigned long long a, unsigned long long b, unsigned& shift,
                                                              unsigned& valid)
{
    const unsigned al = (unsigned)a, ah = (unsigned)(a >> 32), bl = (unsigned)b, bh = (unsigned)(b >> 32);
    const unsigned long long t0 = (unsigned long long)al * bl, t1 = (unsigned long long)al * bh + (t0 >> 32),
                             t2 = (unsigned long long)ah * bl + (unsigned)t1,
                             hi = (unsigned long long)ah * bh + (t1 >> 32) + (t2 >> 32);
    const unsigned hh = (unsigned)(hi >> 32), hl = (unsigned)hi, lh = (unsigned)t2, ll = (unsigned)t0;
    const unsigned sh = ~hh >> 31;
    unsigned long long h = ((unsigned long long)__funnelshift_l(hl, hh, sh) << 32) | __funnelshift_l(lh, hl, sh);
    const unsigned rest = (lh << sh) | ll;
    h += 0x3ff + (rest != 0 ? 1u : ((unsigned)h >> 11) & 1u);
    shift += sh;
    valid &= (unsigned)(h >> 32);
    return h & ~0x7ffull;
}

// ---- products of 64-bit fixed-point numbers ---------------------------------------------------

// v = h 2^32 + l, both signed (|v| < 2^63 - 2^31)
struct Split64 {
    int h, l;
};
__device__ __forceinline__ Split64 split64(long long v)
{
    const int l = (int)v;
    return {(int)(v >> 32) + (int)((unsigned)l >> 31), l};
}

// a b 2^-64 to about one unit: three 32 x 32 -> 64 multiply-adds, the cross terms' high word as it stands in its
// register.  l l' (a quarter of a unit, of either sign) is left out; |h l'| + |h' l| < 2^63.  (Halves of 31 bits need
// shifts for the cross terms and for the result.)
__device__ __forceinline__ long long mul64(Split64 a, Split64 b)
{
    const long long c = (long long)a.l * b.h + ((long long)a.h * b.l + (1ll << 31));
    return (long long)a.h * b.h + (c >> 32);
}

}  // namespace cg
