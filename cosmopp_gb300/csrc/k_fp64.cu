// Plain FP64 path: covariance build, likelihood and adjoint gradient.
//
// build_c_packed and build_c_ref replace CMatrixGenerator::clToCMatrix
// (source/c_matrix_generator.cpp:164-232).  Each thread runs the Bonnet
// recurrence once per pixel pair in registers; the reference restarts it for
// every l (include/legendre.hpp:26-37) but produces the same P_l values bit for
// bit, and the element sum keeps the reference's operation order
//   element += ((clCopy_l * P_l) * B_l) * B_l
// with explicitly rounded (non-fused) FP64 operations, so C is bit-identical
// to the reference's.  build_c_tiled, inside the likelihood, forms the same sum in
// 64-bit fixed point, nearer to the exact value.
//
// The likelihood follows Likelihood::construct / calculate
// (source/likelihood.cpp:69-180): C + N, Cholesky of [C; harmonics, map] (k_digit.cu), ln det
// from the factor's diagonal, chi2 = |L^-1 d|^2; the packed likelihoods keep C^-1 instead.  The
// adjoint gradient (no reference counterpart) is
//   d(-2lnL)/dC_l = sum_ij (C^-1 - a a^T)_ij (2l+1)/(4pi) B_l^2 P_l(x_ij),  a = C^-1 d.
#include <algorithm>
#include <cmath>

#include "cg_fixed.cuh"
#include "cg_internal.h"
#include "cg_launch.cuh"

namespace cg {

namespace {

constexpr double kPi = 3.141592653589793;  // include/math_constants.hpp:8
constexpr int kThreads = 256;
constexpr int kAdjChunk = 48;               // l values accumulated per adjoint pass

// ThreeVector dot (include/three_vector.hpp:37) + clamp (c_matrix_generator.cpp:203-215)
__device__ __forceinline__ double pair_dot(const double* __restrict__ xyz, int N, int i, int j)
{
    double d = __dadd_rn(__dadd_rn(__dmul_rn(xyz[i], xyz[j]), __dmul_rn(xyz[N + i], xyz[N + j])),
                         __dmul_rn(xyz[2 * N + i], xyz[2 * N + j]));
    if (d > 1.0) d = 1.0;
    if (d < -1.0) d = -1.0;
    return d;
}

// sum_{l=2}^{lmax} ((clc_l * P_l) * B_l) * B_l in the reference's order, 4 pairs at once
__device__ __forceinline__ void cmat_sum4(const double x[4], double (&acc)[4], int lmax, const double* sa,
                                          const double* sb, const double* sc, const double* sbeam)
{
    double p0[4], p1[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        p0[q] = 1.0;
        p1[q] = x[q];
        acc[q] = 0.0;
    }
    for (int l = 2; l <= lmax; ++l) {
        const double a = sa[l], b = sb[l], c = sc[l], bm = sbeam[l];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double p = __dsub_rn(__dmul_rn(__dmul_rn(a, x[q]), p1[q]), __dmul_rn(b, p0[q]));
            acc[q] = __dadd_rn(acc[q], __dmul_rn(__dmul_rn(__dmul_rn(c, p), bm), bm));
            p0[q] = p1[q];
            p1[q] = p;
        }
    }
}

__device__ __forceinline__ void load_consts(double* sa, double* sb, double* sc, double* sbeam, int lmax,
                                            const double* lega, const double* legb, const double* beam,
                                            const double* cl)
{
    for (int l = threadIdx.x; l <= lmax; l += blockDim.x) {
        sa[l] = lega[l];
        sb[l] = legb[l];
        sbeam[l] = beam[l];
        // clCopy[l] = cl[l] * (2 l + 1) / (4 pi)   (c_matrix_generator.cpp:190-193)
        sc[l] = (l >= 2) ? __ddiv_rn(__dmul_rn(cl[l], (double)(2 * l + 1)), 4.0 * kPi) : 0.0;
    }
}

// C (+ noise on the diagonal, identity padding) into the tiled layout with the reference's operations, for
// the mixed path's reference point (its FP32 table and factor keep their bits), grid (tiles, B)
__global__ void __launch_bounds__(kThreads) build_c_ref(int n, int N, int lmax, const double* __restrict__ xyz,
                                                          const double* __restrict__ noise,
                                                          const double* __restrict__ lega,
                                                          const double* __restrict__ legb,
                                                          const double* __restrict__ beam,
                                                          const double* __restrict__ cl, int add_noise,
                                                          double* __restrict__ A, size_t strideA)
{
    extern __shared__ double sconst[];
    double* sa = sconst;
    double* sb = sa + (lmax + 1);
    double* sc = sb + (lmax + 1);
    double* sbeam = sc + (lmax + 1);
    const int b = blockIdx.y;
    load_consts(sa, sb, sc, sbeam, lmax, lega, legb, beam, cl + (size_t)b * (lmax + 1));
    __syncthreads();
    int I, J;
    tile_coords(blockIdx.x, I, J);
    double* tile = A + (size_t)b * strideA + (size_t)blockIdx.x * TILE_ELEMS;
    for (int g = 0; g < TILE_ELEMS / (kThreads * 4); ++g) {
        double x[4], v[4];
        int e[4];
        bool real[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            e[q] = threadIdx.x + kThreads * (4 * g + q);
            const int i = I * TS + e[q] % TS, j = J * TS + e[q] / TS;
            real[q] = (i < n && j < n);
            x[q] = real[q] ? pair_dot(xyz, N, i, j) : 0.0;
        }
        cmat_sum4(x, v, lmax, sa, sb, sc, sbeam);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = I * TS + e[q] % TS, j = J * TS + e[q] / TS;
            double val;
            if (real[q]) {
                val = v[q];
                // cInv_(i,j) = c + fiducial(0) + noise  (source/likelihood.cpp:102-110)
                if (add_noise && i == j) val = __dadd_rn(__dadd_rn(val, 0.0), noise[i]);
            } else {
                val = (i == j) ? 1.0 : 0.0;
            }
            tile[e[q]] = val;
        }
    }
}

// ---- covariance for the likelihood, in 64-bit fixed point ----------------------------------
//
// The FP64 pipe gives 2 operations per cycle and SM, the 32 x 32 -> 64 multiply-add 64, and every quantity of
// the Legendre sum is bounded: |P_l| <= 1, |x| <= 1, and the weights w_l = C_l (2l+1)/(4 pi) B_l^2 are
// scaled by a power of two above sum |w_l|.  So the sum runs in integers, x, P_l and w_l with 62 fraction bits, 1 / l
// with 64 (a product drops 64):
//     t = x P_{l-1},  P_l = 2 t - P_{l-2} - (t - P_{l-2}) / l,  S += w_l P_l,
// three multiply-adds a product.  x itself is the dot product of the directions in fixed point, and the
// sum becomes FP64 in integer operations.  The sum is 50 to 200 times nearer to the exact value than the FP64
// recurrence's (lmax 12 to 255).  The P_l are shared by NB batch elements.  The integer pipes bound it (47
// instructions per pair and l with one element, 57 % of the issue slots, 64 % of the multiply-add pipe): one matrix at
// nside 16 2650 us in FP64, 418 with halves of 31 bits, 322 here; sixteen 42 ms, 2.9, 2.3.

// status, the waits' error flag and fixed-point weights of every element: wfix[b][l] = w_l 2^(62 - e), wexp[b] = e with
// sum |w_l| < 2^e; a non-finite weight gives e = kNonFinite and a NaN covariance.  grid B
__global__ void __launch_bounds__(kThreads) legendre_weights(int lmax, const double* __restrict__ beam,
                                                             const double* __restrict__ cl,
                                                             long long* __restrict__ wfix, int* __restrict__ wexp,
                                                             int* __restrict__ status, int* __restrict__ err)
{
    __shared__ double part[kThreads / 32];
    launch_dependents();
    const int b = blockIdx.x, l = threadIdx.x, L1 = lmax + 1;
    const double c = l <= lmax ? cl[(size_t)b * L1 + l] : 0.0;
    // clCopy[l] = cl[l] * (2 l + 1) / (4 pi)   (c_matrix_generator.cpp:190-193)
    double w = 0.0;
    if (l >= 2 && l <= lmax)
        w = __dmul_rn(__dmul_rn(__ddiv_rn(__dmul_rn(c, (double)(2 * l + 1)), 4.0 * kPi), beam[l]), beam[l]);
    double s = fabs(w);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (l % 32 == 0) part[l / 32] = s;
    const int bad = __syncthreads_or(!isfinite(c));
    s = 0.0;
    for (int k = 0; k < kThreads / 32; ++k) s += part[k];
    const int e = isfinite(s) ? (s > 0.0 ? ilogb(s) + 1 : -1000) : kNonFinite;
    if (l <= lmax) wfix[(size_t)b * L1 + l] = e == kNonFinite ? 0 : __double2ll_rn(scalbn(w, 62 - e));
    if (l == 0) {
        wexp[b] = e;
        status[b] = bad ? CG_ERR_NONFINITE : CG_OK;
        if (b == 0) *err = 0;
    }
}

// C (+ noise on the diagonal, identity padding) into the tiled layout; grid (tiles * kBuildParts, ceil(B / NB)), a CTA
// per quarter of a tile, 4 pairs per thread (a CTA per tile left SMs idle: the 55 tiles of nside 8 took 41 us, now 23
// less; the 820 of nside 16, 1.3 waves, 355, now 322).  Directions with a component beyond 1 (a caller's, off the unit
// sphere) take their dot product in FP64, with the reference's clamp.
constexpr int kBuildParts = TILE_ELEMS / (kThreads * 4);

template <int NB>
__global__ void __launch_bounds__(kThreads) build_c_tiled(int n, int N, int lmax, int B,
                                                          const double* __restrict__ xyz,
                                                          const double* __restrict__ noise,
                                                          const long long* __restrict__ wfix,
                                                          const int* __restrict__ wexp, double* __restrict__ A,
                                                          size_t strideA)
{
    extern __shared__ Split64 sfix[];
    __shared__ Split64 dir[2][3][TS];
    const int L1 = lmax + 1, b0 = blockIdx.y * NB;
    wait_prior();
    launch_dependents();       // not before: ext_rows runs beside this without waiting for it
    Split64* sr = sfix;        // 1 / l, l > 2
    Split64* sw = sfix + L1;   // [l][NB]
    const int tix = blockIdx.x / kBuildParts, g = blockIdx.x % kBuildParts;
    int I, J;
    tile_coords(tix, I, J);
    for (int l = threadIdx.x; l <= lmax; l += kThreads) {
        sr[l] = split64(l > 2 ? (long long)((0ull - (unsigned)l) / (unsigned)l + 1) : 0);  // 2^64 / l
#pragma unroll
        for (int q = 0; q < NB; ++q) sw[l * NB + q] = split64(b0 + q < B ? wfix[(size_t)(b0 + q) * L1 + l] : 0);
    }
    bool beyond = false;
    for (int e = threadIdx.x; e < 6 * TS; e += kThreads) {
        const int s = e / (3 * TS), c = e / TS % 3, i = e % TS;
        const double v = xyz[(size_t)c * N + (s ? J : I) * TS + i];
        beyond |= !(fabs(v) <= 1.0);
        dir[s][c][i] = split64(2 * to_fixed<62>(v, 1));
    }
    beyond = __syncthreads_or(beyond);
    Split64 x[4];
    long long p0[4], p1[4], acc[NB][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int e = threadIdx.x + kThreads * (4 * g + q), i = e % TS, j = e / TS;
        long long v = 0;  // with 60 fraction bits
        if (!beyond) {
#pragma unroll
            for (int c = 0; c < 3; ++c) v += mul64(dir[0][c][i], dir[1][c][j]);
            v = 4 * min(max(v, -(1ll << 60)), 1ll << 60);
        } else if (I * TS + i < n && J * TS + j < n) {
            v = 2 * to_fixed<62>(pair_dot(xyz, N, I * TS + i, J * TS + j), 1);
        }
        // P_2 = 2 t - 1 - (t - 1) / 2, t = x^2
        x[q] = split64(v);
        const long long d = 4 * mul64(x[q], x[q]) - (1ll << 62), p = d + (d >> 1) + (1ll << 62);
        p0[q] = v;
        p1[q] = p;
        const Split64 ps = split64(p);
#pragma unroll
        for (int k = 0; k < NB; ++k) acc[k][q] = mul64(ps, sw[2 * NB + k]);
    }
#pragma unroll 2
    for (int l = 3; l <= lmax; ++l) {
        const Split64 rl = sr[l];
        Split64 w[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) w[k] = sw[l * NB + k];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const long long t = 4 * mul64(split64(p1[q]), x[q]), d = t - p0[q];
            const long long p = t + d - mul64(split64(d), rl);
            p0[q] = p1[q];
            p1[q] = p;
            const Split64 ps = split64(p);
#pragma unroll
            for (int k = 0; k < NB; ++k) acc[k][q] += mul64(ps, w[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        if (b0 + k >= B) break;
        const int we = wexp[b0 + k];
        double* tile = A + (size_t)(b0 + k) * strideA + (size_t)tix * TILE_ELEMS;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = threadIdx.x + kThreads * (4 * g + q), i = I * TS + e % TS, j = J * TS + e / TS;
            double val;
            if (i < n && j < n) {
                // a non-finite weight's exponent gives NaN
                val = scaled_int(acc[k][q], we - 60, 0);
                // cInv_(i,j) = c + fiducial(0) + noise  (source/likelihood.cpp:102-110)
                if (i == j) val = __dadd_rn(val, noise[i]);
            } else {
                val = (i == j) ? 1.0 : 0.0;
            }
            tile[e] = val;
        }
    }
}

// Packed output (i <= j at j(j+1)/2 + i) with the reference's operations and rounding, kPairs entries per thread
// of NB elements; grid (ceil(np / (kPairs kThreads)), ceil(B / NB)).
//
// Of the FP64 operations per pair and l, four are the recurrence's, which the elements share, and four each
// element's: ((c P_l) B_l) B_l and the addition.  The FP64 pipe takes a warp instruction every 64 cycles and
// partition, so the three products are formed in integers with the same rounding (some 22 instructions each), the
// final exponents added up beside them.  What is not plainly normal (P_l zero or below 2^-200, a C_l or B_l of 0 or
// an exponent beyond 300 and 150, a product that rounds up to a power of two) goes through the FP64 pipe.
// Four matrices at nside 16: 5.5 ms with all products in the FP64 pipe, 2.4 ms here, that pipe still 81 % busy (B_l's
// partner in the recurrence, b P_(l-2), in integers too: no faster).
constexpr int kPairs = 2;

struct PackedTerm {          // the constants of one l and element
    unsigned long long m;    // significand of c
    double c;
    unsigned k;              // sign and exponent of the product but for P_l's
    int pad;
};
struct PackedL {
    double a, b, bm;
    unsigned long long m;    // significand of bm
    int normal, pad;         // the integer products may be used
};

template <int NB>
__global__ void __launch_bounds__(kThreads) build_c_packed(int n, int N, int lmax, int B, const double* __restrict__ xyz,
                                                           const double* __restrict__ lega,
                                                           const double* __restrict__ legb,
                                                           const double* __restrict__ beam,
                                                           const double* __restrict__ cl, double* __restrict__ out)
{
    extern __shared__ double sconst[];
    PackedL* sl = reinterpret_cast<PackedL*>(sconst);
    PackedTerm* st = reinterpret_cast<PackedTerm*>(sl + lmax + 1);  // [l][NB]
    const int b0 = blockIdx.y * NB;
    auto field = [](double v) { return (int)(((unsigned)__double2hiint(v) >> 20) & 0x7ffu); };
    for (int l = threadIdx.x; l <= lmax; l += kThreads) {
        const double bm = beam[l];
        bool normal = abs(field(bm) - 1023) <= 150;
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            // clCopy[l] = cl[l] * (2 l + 1) / (4 pi)   (c_matrix_generator.cpp:190-193); past B, the last again
            const double c = __ddiv_rn(__dmul_rn(cl[(size_t)min(b0 + k, B - 1) * (lmax + 1) + l], (double)(2 * l + 1)), 4.0 * kPi);
            PackedTerm& t = st[l * NB + k];
            t.c = c;
            t.m = significand(c);
            t.k = ((unsigned)(field(c) + 2 * field(bm) - 3 * 1022 - 1) << 20) + ((unsigned)__double2hiint(c) & 0x80000000u);
            normal = normal && abs(field(c) - 1023) <= 300;
        }
        sl[l] = {lega[l], legb[l], bm, significand(bm), normal, 0};
    }
    __syncthreads();
    const long np = (long)n * (n + 1) / 2;
    const long k0 = kPairs * ((long)blockIdx.x * kThreads + threadIdx.x);
    if (k0 >= np) return;
    long j = (long)((sqrt(8.0 * (double)k0 + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > k0) --j;
    while ((j + 1) * (j + 2) / 2 <= k0) ++j;
    long i = k0 - j * (j + 1) / 2;
    double x[kPairs], p0[kPairs], p1[kPairs], acc[NB][kPairs];
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {  // consecutive packed entries: walk i, wrap to the next column
        x[q] = (k0 + q < np) ? pair_dot(xyz, N, (int)i, (int)j) : 0.0;
        if (++i > j) { ++j; i = 0; }
        p0[q] = 1.0;
        p1[q] = x[q];
#pragma unroll
        for (int k = 0; k < NB; ++k) acc[k][q] = 0.0;
    }
    for (int l = 2; l <= lmax; ++l) {
        const PackedL c = sl[l];
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
            const double p = __dsub_rn(__dmul_rn(__dmul_rn(c.a, x[q]), p1[q]), __dmul_rn(c.b, p0[q]));
            p0[q] = p1[q];
            p1[q] = p;
            const unsigned ph = (unsigned)__double2hiint(p);
            const unsigned long long pm = significand(p);
            double v[NB];
            unsigned valid = 0xffffffffu;
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const PackedTerm& t = st[l * NB + k];
                unsigned shift = 0;
                const unsigned long long m =
                    mul_significand(mul_significand(mul_significand(pm, t.m, shift, valid), c.m, shift, valid), c.m, shift, valid);
                v[k] = __hiloint2double((int)((unsigned)(m >> 43) + (ph & 0xfff00000u) + t.k - (shift << 20)), (int)(unsigned)(m >> 11));
            }
            if (!c.normal || (int)valid >= 0 || (ph & 0x7ff00000u) - (823u << 20) > (201u << 20)) {
#pragma unroll
                for (int k = 0; k < NB; ++k) v[k] = __dmul_rn(__dmul_rn(__dmul_rn(st[l * NB + k].c, p), c.bm), c.bm);
            }
#pragma unroll
            for (int k = 0; k < NB; ++k) acc[k][q] = __dadd_rn(acc[k][q], v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < NB; ++k)
        if (b0 + k < B)
#pragma unroll
            for (int q = 0; q < kPairs; ++q)
                if (k0 + q < np) out[(size_t)(b0 + k) * np + k0 + q] = acc[k][q];
}

// CMatrixGenerator::getFiducialMatrix (source/c_matrix_generator.cpp:706-772), packed i <= j:
//   element = sum_{l=lo}^{hi} (((fc_l * P_l) * B_l) * B_l) + (((m0 * (1 + x)) * B_2) * B_2)
// with fc_l = cl_l * ((2l+1)/(4 pi)) and m0 = 100 cl_2 formed on the host as the reference
// forms them; tab = [a | b | fc | beam], hi + 1 entries each; lo >= 2.
__global__ void __launch_bounds__(kThreads) build_fid_packed(int n, int N, int lo, int hi,
                                                             const double* __restrict__ xyz,
                                                             const double* __restrict__ tab, double m0,
                                                             double* __restrict__ out)
{
    extern __shared__ double sconst[];
    const int L1 = hi + 1;
    for (int e = threadIdx.x; e < 4 * L1; e += blockDim.x) sconst[e] = tab[e];
    __syncthreads();
    const double* sa = sconst;
    const double* sb = sa + L1;
    const double* sf = sb + L1;
    const double* sbeam = sf + L1;
    const long np = (long)n * (n + 1) / 2;
    const long k0 = 4 * ((long)blockIdx.x * kThreads + threadIdx.x);
    if (k0 >= np) return;
    long j = (long)((sqrt(8.0 * (double)k0 + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > k0) --j;
    while ((j + 1) * (j + 2) / 2 <= k0) ++j;
    long i = k0 - j * (j + 1) / 2;
    double x[4], p0[4], p1[4], acc[4];
    long kk[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        kk[q] = k0 + q;
        x[q] = (kk[q] < np) ? pair_dot(xyz, N, (int)i, (int)j) : 0.0;
        if (++i > j) { ++j; i = 0; }
        p0[q] = 1.0;
        p1[q] = x[q];
        acc[q] = 0.0;
    }
    for (int l = 2; l < lo; ++l) {  // recurrence only (include/legendre.hpp:34)
        const double a = sa[l], b = sb[l];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double p = __dsub_rn(__dmul_rn(__dmul_rn(a, x[q]), p1[q]), __dmul_rn(b, p0[q]));
            p0[q] = p1[q];
            p1[q] = p;
        }
    }
    for (int l = lo; l <= hi; ++l) {
        const double a = sa[l], b = sb[l], f = sf[l], bm = sbeam[l];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double p = __dsub_rn(__dmul_rn(__dmul_rn(a, x[q]), p1[q]), __dmul_rn(b, p0[q]));
            acc[q] = __dadd_rn(acc[q], __dmul_rn(__dmul_rn(__dmul_rn(f, p), bm), bm));
            p0[q] = p1[q];
            p1[q] = p;
        }
    }
    const double b2 = sbeam[2];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (kk[q] < np)
            out[kk[q]] = __dadd_rn(acc[q], __dmul_rn(__dmul_rn(__dmul_rn(m0, __dadd_rn(1.0, x[q])), b2), b2));
}

// An element without a number: a C_l that is none, whose covariance the factorisation puts benign values in place of,
// or a bounded wait that gave up.  Its outputs are NaN, asked for its status or not.  (status, err nullable)
__device__ __forceinline__ bool no_number(const int* __restrict__ status, const int* __restrict__ err, int b)
{
    return status && (status[b] == CG_ERR_NONFINITE || *err);
}
__device__ __forceinline__ double nan_value() { return __longlong_as_double(0x7ff8000000000000ll); }

// ln det = 2 sum_i ln L_ii over the n real pixels (source/matrix_impl.cpp:322-338), grid B
// (an FP64 logarithm is some 30 instructions of 64 cycles each and partition)
constexpr int kLogThreads = 1024;
__global__ void __launch_bounds__(kLogThreads) logdet_reduce(int n, int N, const double* __restrict__ diag,
                                                             const int* __restrict__ status, const int* __restrict__ err,
                                                             double* __restrict__ logdet)
{
    launch_dependents();
    wait_prior();
    __shared__ double red[kLogThreads];
    const int b = blockIdx.x;
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kLogThreads) s += log(fabs(diag[(size_t)b * N + i]));
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kLogThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) logdet[b] = no_number(status, err, b) ? nan_value() : 2.0 * red[0];
}

// padded copy of the data maps into dvec[b][N]
__global__ void pad_data(int n, int N, int B, const double* __restrict__ d, int d_stride, double* __restrict__ dv)
{
    const int b = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N || b >= B) return;
    dv[(size_t)b * N + i] = (i < n) ? d[(size_t)b * d_stride + i] : 0.0;
}

// alpha = V d with V symmetric in lower tiles; grid (nt, B); thread (row r, part q)
template <typename T>
__global__ void __launch_bounds__(kThreads) symv_tiled(int nt, int N, const T* __restrict__ V, size_t strideA,
                                                       const double* __restrict__ dv, double* __restrict__ alpha)
{
    __shared__ double part[4][TS];
    const int I = blockIdx.x, b = blockIdx.y;
    const int r = threadIdx.x % TS, q = threadIdx.x / TS;
    const T* Vb = V + (size_t)b * strideA;
    const double* db = dv + (size_t)b * N;
    double s = 0.0;
    for (int J = 0; J < nt; ++J) {
        if (J <= I) {
            const T* t = Vb + (size_t)tile_index(I, J) * TILE_ELEMS;
            for (int c = q; c < TS; c += 4) s += (double)t[r + TS * c] * db[J * TS + c];
        } else {
            const T* t = Vb + (size_t)tile_index(J, I) * TILE_ELEMS;
            for (int c = q; c < TS; c += 4) s += (double)t[c + TS * r] * db[J * TS + c];
        }
    }
    part[q][r] = s;
    __syncthreads();
    if (q == 0) alpha[(size_t)b * N + I * TS + r] = ((part[0][r] + part[1][r]) + part[2][r]) + part[3][r];
}

// chi2 = d . alpha, m2lnl = chi2 + logdet; grid B
__global__ void __launch_bounds__(kThreads) chi2_finish(int n, int N, const double* __restrict__ dv,
                                                        const double* __restrict__ alpha,
                                                        const double* __restrict__ logdet, const int* __restrict__ status,
                                                        const int* __restrict__ err, double* __restrict__ m2lnl,
                                                        double* __restrict__ chi2)
{
    __shared__ double red[kThreads];
    const int b = blockIdx.x;
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kThreads) s += dv[(size_t)b * N + i] * alpha[(size_t)b * N + i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double x = no_number(status, err, b) ? nan_value() : red[0];
        if (chi2) chi2[b] = x;
        m2lnl[b] = x + logdet[b];
    }
}

// Adjoint partial sums: for every lower tile, sum over its pairs of
// w_ij P_l(x_ij) for l in [l0, l1), w_ij = mult (V_ij - a_i a_j); grid (tiles, B)
__global__ void __launch_bounds__(kThreads) adjoint_tiles(int n, int N, int l0, int l1, const double* __restrict__ xyz,
                                                          const double* __restrict__ lega,
                                                          const double* __restrict__ legb,
                                                          const double* __restrict__ V, size_t strideA,
                                                          const double* __restrict__ alpha,
                                                          double* __restrict__ gpart, int ntile, int lstride)
{
    __shared__ double sa[256], sb[256];
    __shared__ double red[kThreads / 32][kAdjChunk];
    for (int l = threadIdx.x; l < l1 && l < 256; l += kThreads) { sa[l] = lega[l]; sb[l] = legb[l]; }
    __syncthreads();
    int I, J;
    tile_coords(blockIdx.x, I, J);
    const int b = blockIdx.y;
    const double* tile = V + (size_t)b * strideA + (size_t)blockIdx.x * TILE_ELEMS;
    const double* al = alpha + (size_t)b * N;
    double acc[kAdjChunk];
#pragma unroll
    for (int c = 0; c < kAdjChunk; ++c) acc[c] = 0.0;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) {
        const int i = I * TS + e % TS, j = J * TS + e / TS;
        if (i >= n || j >= n || j > i) continue;
        const double w = (i == j ? 1.0 : 2.0) * (tile[e] - al[i] * al[j]);
        const double x = pair_dot(xyz, N, i, j);
        double p0 = 1.0, p1 = x;
        for (int l = 2; l < l0; ++l) {  // advance to P_{l0-1}, P_{l0-2}
            const double p = (sa[l] * x) * p1 - sb[l] * p0;
            p0 = p1;
            p1 = p;
        }
#pragma unroll
        for (int c = 0; c < kAdjChunk; ++c) {
            const int l = l0 + c;
            if (l < l1) {
                const double p = (sa[l] * x) * p1 - sb[l] * p0;
                acc[c] += w * p;
                p0 = p1;
                p1 = p;
            }
        }
    }
    // deterministic block reduction: warp shuffles, then warps in order
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
#pragma unroll
    for (int c = 0; c < kAdjChunk; ++c) {
        double v = acc[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][c] = v;
    }
    __syncthreads();
    if (threadIdx.x < kAdjChunk && l0 + (int)threadIdx.x < l1) {
        double s = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) s += red[w][threadIdx.x];
        gpart[((size_t)b * ntile + blockIdx.x) * lstride + l0 + threadIdx.x] = s;
    }
}

// grad_l = (sum over tiles) * ((2l+1)/(4 pi)) * B_l * B_l; grid B
__global__ void adjoint_finish(int lmax, int ntile, const double* __restrict__ gpart, const double* __restrict__ beam,
                               const int* __restrict__ status, const int* __restrict__ err, double* __restrict__ grad)
{
    const int b = blockIdx.x;
    const bool none = no_number(status, err, b);
    for (int l = threadIdx.x; l <= lmax; l += blockDim.x) {
        double s = 0.0;
        if (l >= 2)
            for (int t = 0; t < ntile; ++t) s += gpart[((size_t)b * ntile + t) * (lmax + 1) + l];
        grad[(size_t)b * (lmax + 1) + l] = (l < 2) ? 0.0 : none ? nan_value() : s * ((2 * l + 1) / (4 * kPi)) * beam[l] * beam[l];
    }
}

// a bounded device wait that gave up (*err) marks every element of the batch
__global__ void copy_status(int B, const int* __restrict__ src, const int* __restrict__ err, int* __restrict__ dst)
{
    launch_dependents();
    wait_prior();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < B) dst[b] = *err ? CG_ERR_TIMEOUT : src[b];
}

// A = c + fid + noise from packed host-layout arrays into the tiled layout,
// in the reference's summation order (source/likelihood.cpp:102-110); grid tiles
__global__ void __launch_bounds__(kThreads) packed_sum_to_tiled(int n, const double* __restrict__ c,
                                                                const double* __restrict__ f,
                                                                const double* __restrict__ nz, double* __restrict__ A,
                                                                int* __restrict__ bad)
{
    int I, J;
    tile_coords(blockIdx.x, I, J);
    double* tile = A + (size_t)blockIdx.x * TILE_ELEMS;
    bool nonfinite = false;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) {
        const int i = I * TS + e % TS, j = J * TS + e / TS;
        double v;
        if (i < n && j < n) {
            const int lo = i < j ? i : j, hi = i < j ? j : i;
            const size_t k = (size_t)hi * (hi + 1) / 2 + lo;
            const double ck = c[k], fk = f ? f[k] : 0.0, nk = nz ? nz[k] : 0.0;
            nonfinite |= !(isfinite(ck) && isfinite(fk) && isfinite(nk));
            v = __dadd_rn(__dadd_rn(ck, fk), nk);
        } else {
            v = (i == j) ? 1.0 : 0.0;
        }
        tile[e] = v;
    }
    if (nonfinite && bad) *bad = 1;
}

__global__ void dot_kernel(int n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out)
{
    __shared__ double red[kThreads];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kThreads) s += a[i] * b[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// The quadratic forms of the packed Likelihood from its inverse's lower tiles: part[t][0] = t^T V t and, with a
// foreground f, part[t][1] = t^T V f, part[t][2] = f^T V f over tile t and its mirror.  One CTA per tile: the
// matrix is read once for both vectors and every SM takes part (a CTA per row block and vector left 40 SMs to
// do it, 152 us a vector at 2469 pixels); a tile costs half the products of a matrix-vector product, whose
// vector nobody needs.  grid tiles
__global__ void __launch_bounds__(kThreads) quad_tiles(const double* __restrict__ V, const double* __restrict__ tv,
                                                       const double* __restrict__ fv, double* __restrict__ part)
{
    __shared__ double red[2][4][TS];
    __shared__ double sum[3][2];
    int I, J;
    tile_coords(blockIdx.x, I, J);
    const double* tile = V + (size_t)blockIdx.x * TILE_ELEMS;
    const int r = threadIdx.x % TS, q = threadIdx.x / TS;
    double y = 0.0, z = 0.0;
#pragma unroll
    for (int c = q; c < TS; c += 4) {
        const double v = tile[r + TS * c];
        y = fma(v, tv[J * TS + c], y);
        if (fv) z = fma(v, fv[J * TS + c], z);
    }
    red[0][q][r] = y;
    red[1][q][r] = z;
    __syncthreads();
    if (threadIdx.x < TS) {
        y = ((red[0][0][r] + red[0][1][r]) + red[0][2][r]) + red[0][3][r];
        z = ((red[1][0][r] + red[1][1][r]) + red[1][2][r]) + red[1][3][r];
        const double t = tv[I * TS + r], f = fv ? fv[I * TS + r] : 0.0, two = I == J ? 1.0 : 2.0;
        double s[3] = {two * (t * y), I == J ? t * z : fma(t, z, f * y), two * (f * z)};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], o);
            if (r % 32 == 0) sum[k][r / 32] = s[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) part[3 * (size_t)blockIdx.x + threadIdx.x] = sum[threadIdx.x][0] + sum[threadIdx.x][1];
}

// out[k] = sum over tiles of part[t][k]; grid 3
__global__ void __launch_bounds__(kThreads) quad_sum(int ntile, const double* __restrict__ part,
                                                     double* __restrict__ out)
{
    __shared__ double red[kThreads];
    double s = 0.0;
    for (int t = threadIdx.x; t < ntile; t += kThreads) s += part[3 * (size_t)t + blockIdx.x];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// Dense FP64 helpers of the polarisation likelihood's set-up (row-major, leading dimension
// ld, a multiple of 128, zero padding beyond n; the products run in k_digit.cu on 64 x 64 tiles).

// row-major to tiles (I, J) at I nt + J, element (r, c) at r + 64 c; grid (nt, nt)
__global__ void __launch_bounds__(kThreads) dense_to_tiles(int ld, const double* __restrict__ d, double* __restrict__ t)
{
    const int I = blockIdx.x, J = blockIdx.y, nt = ld / TS;
    double* tile = t + ((size_t)I * nt + J) * TILE_ELEMS;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads)
        tile[e % TS * TS + e / TS] = d[(size_t)(I * TS + e / TS) * ld + J * TS + e % TS];
}

// packed symmetric (i <= j at j(j+1)/2 + i) to dense, zero outside n x n; grid covers ld x ld
__global__ void packed_to_dense(int n, int ld, const double* __restrict__ pk, double* __restrict__ d)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)ld * ld) return;
    const int r = (int)(e % ld), c = (int)(e / ld);
    const int i = min(r, c), j = max(r, c);
    d[e] = (j < n) ? pk[(size_t)j * (j + 1) / 2 + i] : 0.0;
}

// the upper triangle of a symmetric matrix in tiles, packed
__global__ void tiles_to_packed(int n, int nt, const double* __restrict__ t, double* __restrict__ pk)
{
    const long np = (long)n * (n + 1) / 2;
    const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= np) return;
    long j = (long)((sqrt(8.0 * (double)k + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > k) --j;
    while ((j + 1) * (j + 2) / 2 <= k) ++j;
    const long i = k - j * (j + 1) / 2;
    pk[k] = t[((size_t)(i / TS) * nt + j / TS) * TILE_ELEMS + i % TS + TS * (j % TS)];
}

// w = v - N s, a warp per row: 32 partial sums over its columns, then a tree (one thread per row left five CTAs
// to do it, 287 us at 1228 rows)
__global__ void __launch_bounds__(kThreads) dense_residual(int n, int ld, const double* __restrict__ Nm,
                                                           const double* __restrict__ v, const double* __restrict__ sv,
                                                           double* __restrict__ w)
{
    const int i = blockIdx.x * (kThreads / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (i >= n) return;
    double acc = 0.0;
    for (int j = lane; j < n; j += 32) acc = fma(Nm[(size_t)i * ld + j], sv[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) w[i] = v[i] - acc;
}

// LegendrePolynomialContainer's table (source/c_matrix_generator.cpp:30-76): P_l(x_ij) for
// l0 <= l < l1 at out[(l - l0) np + j(j+1)/2 + i], i <= j, by Math::Legendre's recurrence
// (include/legendre.hpp:26-37: P_0 = 1, P_1 = x, P_l = ((2 - 1/l) x) P_{l-1} - (1 - 1/l) P_{l-2},
// coefficients a_l, b_l from the host) with the reference's dot product and clamp, so the
// table is bit-identical.  One thread per pair; stores of one l are coalesced over pairs.
__global__ void __launch_bounds__(kThreads) legendre_table(int n, int N, int l0, int l1,
                                                           const double* __restrict__ xyz,
                                                           const double* __restrict__ a,
                                                           const double* __restrict__ b,
                                                           double* __restrict__ out)
{
    const long np = (long)n * (n + 1) / 2;
    const long k = (long)blockIdx.x * kThreads + threadIdx.x;
    if (k >= np) return;
    long j = (long)((sqrt(8.0 * (double)k + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > k) --j;
    while ((j + 1) * (j + 2) / 2 <= k) ++j;
    const int i = (int)(k - j * (j + 1) / 2);
    const double x = pair_dot(xyz, N, i, (int)j);
    double p0 = 1.0, p1 = x;
    for (int l = 0; l < l1; ++l) {
        double p;
        if (l == 0) {
            p = 1.0;
        } else if (l == 1) {
            p = x;
        } else {
            p = __dsub_rn(__dmul_rn(__dmul_rn(a[l], x), p1), __dmul_rn(b[l], p0));
            p0 = p1;
            p1 = p;
        }
        if (l >= l0) out[(size_t)(l - l0) * np + k] = p;
    }
}

// Averaging step of CMatrixGenerator::calculateNoiseMatrix (source/c_matrix_generator.cpp:887-910):
// N_ij = (sum_k s_k[i] s_k[j]) / nsims, k in order, every product and sum rounded on its own
// (the reference's loop, compiled without contraction), so the packed result is
// bit-identical.  A CTA computes one 64x64 tile (I <= J) of the upper triangle; 16-deep
// slices of the two 64-pixel panels are staged in shared memory; each thread keeps a
// 4x4 block of sums at rows ty + 16a and columns tx + 16b.
constexpr int kNoiseT = 64, kNoiseK = 16;

__global__ void __launch_bounds__(kThreads, 2) noise_syrk_packed(int nsims, int n, const double* __restrict__ sims,
                                                              double* __restrict__ out)
{
    const long t = blockIdx.x;
    int J = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((long)J * (J + 1) / 2 > t) --J;
    while ((long)(J + 1) * (J + 2) / 2 <= t) ++J;
    const int I = (int)(t - (long)J * (J + 1) / 2);
    __shared__ double si[kNoiseK][kNoiseT], sj[kNoiseK][kNoiseT];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    for (int k0 = 0; k0 < nsims; k0 += kNoiseK) {
#pragma unroll
        for (int r = 0; r < kNoiseK * kNoiseT / kThreads; ++r) {
            const int e = threadIdx.x + r * kThreads, kk = e / kNoiseT, c = e % kNoiseT, k = k0 + kk;
            const int gi = I * kNoiseT + c, gj = J * kNoiseT + c;
            si[kk][c] = (k < nsims && gi < n) ? sims[(size_t)k * n + gi] : 0.0;
            sj[kk][c] = (k < nsims && gj < n) ? sims[(size_t)k * n + gj] : 0.0;
        }
        __syncthreads();
        const int kend = min(kNoiseK, nsims - k0);
        for (int kk = 0; kk < kend; ++kk) {
            double x[4], y[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) x[a] = si[kk][ty + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) y[b] = sj[kk][tx + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = __dadd_rn(acc[a][b], __dmul_rn(x[a], y[b]));
        }
        __syncthreads();
    }
    const double dn = (double)nsims;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = I * kNoiseT + ty + 16 * a, j = J * kNoiseT + tx + 16 * b;
            if (i <= j && j < n) out[(size_t)j * (j + 1) / 2 + i] = __ddiv_rn(acc[a][b], dn);
        }
}

// per-pixel mean over the simulations, summed in order (source/c_matrix_generator.cpp:901-910)
__global__ void sim_means(int nsims, int n, const double* __restrict__ sims, double* __restrict__ mean)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double s = 0.0;
    for (int k = 0; k < nsims; ++k) s = __dadd_rn(s, sims[(size_t)k * n + j]);
    mean[j] = __ddiv_rn(s, (double)nsims);
}

// E = identity of DIGIT_EXT_IDENTITY: tile (eb, k) at tile_index(k, eb); grid (tiles, B)
__global__ void __launch_bounds__(kThreads) identity_rows(double* __restrict__ E, size_t strideE)
{
    int k, eb;
    tile_coords(blockIdx.x, k, eb);
    double* tile = E + (size_t)blockIdx.y * strideE + (size_t)blockIdx.x * TILE_ELEMS;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) tile[e] = (k == eb && e % TS == e / TS) ? 1.0 : 0.0;
}

// the harmonics' rows [h][N] as E's tiles (eb, k), zero beyond nharm; grid (nt, ne)
__global__ void __launch_bounds__(kThreads) harmonic_tiles(int N, int nt, int nharm, const double* __restrict__ Y,
                                                           double* __restrict__ Yt)
{
    __shared__ double s[TS][TS + 1];
    const int k = blockIdx.x, eb = blockIdx.y;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) {
        const int c = e % TS, r = e / TS, h = eb * TS + r;
        s[r][c] = h < nharm ? Y[(size_t)h * N + k * TS + c] : 0.0;
    }
    __syncthreads();
    double* tile = Yt + ((size_t)eb * nt + k) * TILE_ELEMS;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) tile[e] = s[e % TS][e / TS];
}

// E's rows at the start: the harmonics (Yt, nullable) and the map as row drow; grid (nt, ne, B)
__global__ void __launch_bounds__(kThreads) ext_rows(int n, int nt, int drow, const double* __restrict__ Yt,
                                                     const double* __restrict__ d, int d_stride,
                                                     double* __restrict__ E, size_t strideE)
{
    launch_dependents();
    const int k = blockIdx.x, eb = blockIdx.y, b = blockIdx.z;
    const size_t off = ((size_t)eb * nt + k) * TILE_ELEMS;
    double* tile = E + (size_t)b * strideE + off;
    const int rd = drow - eb * TS;
    for (int e = threadIdx.x; e < TILE_ELEMS; e += kThreads) {
        double v = Yt ? Yt[off + e] : 0.0;
        if (e % TS == rd) {
            const int i = k * TS + e / TS;
            v = i < n ? d[(size_t)b * d_stride + i] : 0.0;
        }
        tile[e] = v;
    }
    wait_prior();  // the covariance, for the kernels after this one
}

// y = L^-1 d from E's row drow, chi2 = y . y, m2lnl = chi2 + logdet; grid B
__global__ void __launch_bounds__(kThreads) chi2_rows(int nt, int drow, const double* __restrict__ E, size_t strideE,
                                                      const double* __restrict__ logdet, const int* __restrict__ status,
                                                      const int* __restrict__ err, double* __restrict__ y,
                                                      double* __restrict__ m2lnl, double* __restrict__ chi2,
                                                      double* __restrict__ logdet_out)
{
    launch_dependents();
    wait_prior();
    __shared__ double red[kThreads];
    const int b = blockIdx.x, N = nt * TS;
    const double* Eb = E + (size_t)b * strideE + (size_t)(drow / TS) * nt * TILE_ELEMS + drow % TS;
    double s = 0.0;
    for (int i = threadIdx.x; i < N; i += kThreads) {
        const double v = Eb[(size_t)i * TS];  // tile i / 64, column i % 64: consecutive columns of the block row
        y[(size_t)b * N + i] = v;
        s = fma(v, v, s);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double x = no_number(status, err, b) ? nan_value() : red[0];
        if (chi2) chi2[b] = x;
        if (logdet_out) logdet_out[b] = logdet[b];
        m2lnl[b] = x + logdet[b];
    }
}

// Gradient through the harmonics: with Z = L^-1 Y (Y_l the 2l + 1 harmonics of l times B_l at the
// pixels, dC/dC_l = Y_l Y_l^T by the addition theorem) and y = L^-1 d,
//   d(-2lnL)/dC_l = tr(C^-1 Y_l Y_l^T) - |Y_l^T C^-1 d|^2 = sum_{h in l} (|Z_h|^2 - (Z_h . y)^2).
// part[b][z][0 / 1][h] = the sums over block columns k = z, z + kHarmSplit, ...; grid (ne, kHarmSplit, B)
constexpr int kHarmSplit = 8;
__global__ void __launch_bounds__(kThreads) harmonic_sums(int nt, int ne, const double* __restrict__ E, size_t strideE,
                                                          const double* __restrict__ y, double* __restrict__ part)
{
    launch_dependents();
    wait_prior();
    __shared__ double red[2][4][TS];
    const int eb = blockIdx.x, z = blockIdx.y, b = blockIdx.z, r = threadIdx.x % TS, q = threadIdx.x / TS;
    const double* Eb = E + (size_t)b * strideE + (size_t)eb * nt * TILE_ELEMS;
    const double* yb = y + (size_t)b * nt * TS;
    double zz = 0.0, zy = 0.0;
    for (int k = z; k < nt; k += kHarmSplit)
#pragma unroll 8
        for (int c = q; c < TS; c += 4) {
            const double v = Eb[(size_t)k * TILE_ELEMS + r + TS * c];
            zz = fma(v, v, zz);
            zy = fma(v, yb[k * TS + c], zy);
        }
    red[0][q][r] = zz;
    red[1][q][r] = zy;
    __syncthreads();
    if (q < 2) {
        const size_t nh = (size_t)ne * TS;
        part[(((size_t)b * kHarmSplit + z) * 2 + q) * nh + eb * TS + r] =
            ((red[q][0][r] + red[q][1][r]) + red[q][2][r]) + red[q][3][r];
    }
}

// grad_l from the sums, a warp per l; grid (ceil((lmax + 1) / 8), B)
__global__ void __launch_bounds__(kThreads) harmonic_grad(int lmax, int ne, const double* __restrict__ part,
                                                          const int* __restrict__ status, const int* __restrict__ err,
                                                          double* __restrict__ grad)
{
    launch_dependents();
    wait_prior();
    const int b = blockIdx.y, l = blockIdx.x * (kThreads / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (l > lmax) return;
    const size_t nh = (size_t)ne * TS;
    const double* p = part + (size_t)b * kHarmSplit * 2 * nh;
    double g = 0.0;
    if (l >= 2)
        for (int h = l * l - 4 + lane; h < (l + 1) * (l + 1) - 4; h += 32) {
            double zz = 0.0, zy = 0.0;
            for (int z = 0; z < kHarmSplit; ++z) {
                zz += p[(size_t)(2 * z) * nh + h];
                zy += p[(size_t)(2 * z + 1) * nh + h];
            }
            g += zz - zy * zy;
        }
    for (int o = 16; o > 0; o >>= 1) g += __shfl_down_sync(0xffffffffu, g, o);
    if (lane == 0) grad[(size_t)b * (lmax + 1) + l] = l >= 2 && no_number(status, err, b) ? nan_value() : g;
}

}  // namespace

void fp64_packed_to_tiled(int n, int nt, const double* c, const double* f, const double* nz, double* A, int* bad,
                          cudaStream_t s)
{
    packed_sum_to_tiled<<<ntiles_lower(nt), kThreads, 0, s>>>(n, c, f, nz, A, bad);
}

void fp64_symv(int B, int nt, int N, const double* V, const double* dv, double* alpha, cudaStream_t s)
{
    symv_tiled<double><<<dim3(nt, B), kThreads, 0, s>>>(nt, N, V, tiled_elems(nt), dv, alpha);
}

void fp64_quad(int nt, const double* V, const double* tv, const double* fv, double* part, double* out, cudaStream_t s)
{
    quad_tiles<<<ntiles_lower(nt), kThreads, 0, s>>>(V, tv, fv, part);
    quad_sum<<<fv ? 3 : 1, kThreads, 0, s>>>(ntiles_lower(nt), part, out);
}

void fp64_logdet(int B, int n, int N, const double* diag, double* out, cudaStream_t s)
{
    logdet_reduce<<<B, kLogThreads, 0, s>>>(n, N, diag, nullptr, nullptr, out);
}

void fp64_dot(int n, const double* a, const double* b, double* out, cudaStream_t s)
{
    dot_kernel<<<1, kThreads, 0, s>>>(n, a, b, out);
}

void fp64_free(cg_ctx* ctx)
{
    Fp64Work& w = ctx->w64;
    cudaFree(w.A); cudaFree(w.E); cudaFree(w.dig); cudaFree(w.diag); cudaFree(w.dvec);
    cudaFree(w.alpha); cudaFree(w.gpart); cudaFree(w.st); cudaFree(w.ld); cudaFree(w.err);
    cudaFree(w.wfix); cudaFree(w.wexp);
    w = Fp64Work();
}

static int nharm_of(int lmax) { return (lmax + 1) * (lmax + 1) - 4; }  // l = 2..lmax

// The factorisation's extra block rows (even): the map alone for a value, the harmonics and the map
// for a gradient, the identity where the gradient goes through C^-1
static int ext_blocks(const cg_ctx* ctx, bool grad)
{
    if (grad && !ctx->harm) return ctx->nt;
    const int rows = grad ? nharm_of(ctx->lmax) + 1 : 1;
    return 2 * ((rows + 2 * TS - 1) / (2 * TS));
}

// Doubles of E per element, for the larger of a value's and a gradient's rows (the identity of two block rows is three
// tiles, the map's 128 rows four)
static size_t ext_elems(const cg_ctx* ctx)
{
    auto rows = [&](bool grad) { return (size_t)ext_blocks(ctx, grad) * ctx->nt * TILE_ELEMS; };
    return ctx->harm ? rows(true) : std::max(rows(false), tiled_elems(ctx->nt));
}

static size_t gpart_elems(const cg_ctx* ctx)
{
    return ctx->harm ? (size_t)kHarmSplit * 2 * ext_blocks(ctx, true) * TS
                     : (size_t)ntiles_lower(ctx->nt) * (ctx->lmax + 1);
}

// The harmonics' route takes nh / 128 block-row pairs through every column of the factorisation, the
// route through C^-1 about 2/3 of the matrix's own pairs and then (lmax - 1) FP64 recurrence steps per
// pixel pair, 0.8 lmax pairs' worth of time.  The addition theorem needs unit directions: what |v|^2
// lacks to 1 puts the gradient off by l (l + 1) / 2 times that.  cg_pix2vec's are unit vectors; a caller's are taken as
// such below 1e-15, which leaves what rounding does to a normalised vector (6.7e-16 at most in 3 million of five
// kinds) and stays within the rounding of the dot products (with the line at 1e-14 the gradient's error at l = 60 was
// 8e-13 of its terms, 5e-15 through C^-1).
bool fp64_harmonics_ok(int n, int nt, int lmax, const double* xyz)
{
    if ((double)nharm_of(lmax) / 128.0 > nt / 3.0 + 0.8 * lmax) return false;
    if (xyz)
        for (int i = 0; i < n; ++i) {
            const double x = xyz[3 * (size_t)i], y = xyz[3 * (size_t)i + 1], z = xyz[3 * (size_t)i + 2];
            if (!(fabs(x * x + y * y + z * z - 1.0) <= 1e-15)) return false;
        }
    return true;
}

// The allocations of fp64_ensure
void fp64_bytes(const cg_ctx* ctx, size_t* fixed, size_t* per_element)
{
    *fixed = sizeof(int) + (ctx->harm ? sizeof(double) * ext_elems(ctx) : 0);
    *per_element = sizeof(double) * (tiled_elems(ctx->nt) + ext_elems(ctx) + 3 * (size_t)ctx->N +
                                     gpart_elems(ctx) + 1) +
                   sizeof(long long) * ((size_t)ctx->lmax + 1) + 2 * sizeof(int) + digit_bytes(ctx->nt, ext_blocks(ctx, true));
}

// The workspace of B elements, for values and gradients alike, so that it moves only when B grows: a call may be
// captured after any call of as many elements, and a captured one stays valid through every later call of no more.
static int fp64_ensure(cg_ctx* ctx, int B)
{
    Fp64Work& w = ctx->w64;
    if (w.cap >= B) return CG_OK;
    const size_t n = B;
    fp64_free(ctx);
    auto alloc = [](auto** p, size_t count) { return cudaMalloc((void**)p, sizeof(**p) * count) == cudaSuccess; };
    w.ext_elems = ext_elems(ctx);
    if (!(alloc(&w.A, tiled_elems(ctx->nt) * n) && alloc(&w.E, w.ext_elems * (n + (ctx->harm ? 1 : 0))) &&
          alloc(&w.dig, digit_bytes(ctx->nt, ext_blocks(ctx, true)) * n) && alloc(&w.diag, ctx->N * n) &&
          alloc(&w.dvec, ctx->N * n) && alloc(&w.alpha, ctx->N * n) && alloc(&w.gpart, gpart_elems(ctx) * n) &&
          alloc(&w.st, n) && alloc(&w.ld, n) && alloc(&w.wfix, (ctx->lmax + 1) * n) && alloc(&w.wexp, n) &&
          alloc(&w.err, 1))) {
        fp64_free(ctx);
        cudaGetLastError();
        ctx->err = "device allocation failed for the FP64 workspace";
        return CG_ERR_ALLOC;
    }
    w.Yt = ctx->harm ? w.E + w.ext_elems * n : nullptr;
    w.cap = B;
    return CG_OK;
}

// The harmonics of the pixels in Yt, by the first gradient call on a workspace (in its stream, by way of E, which the
// call fills afterwards; a captured call carries them along, and they count as made only when they were run)
static int fp64_harmonics(cg_ctx* ctx, cudaStream_t s)
{
    Fp64Work& w = ctx->w64;
    if (w.have_yt) return CG_OK;
    if (int rc = ylm_fill(ctx, w.E, s)) return rc;
    harmonic_tiles<<<dim3(ctx->nt, ext_blocks(ctx, true)), kThreads, 0, s>>>(ctx->N, ctx->nt, nharm_of(ctx->lmax), w.E, w.Yt);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    w.have_yt = cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return CG_OK;
}

int fp64_identity_rows(cg_ctx* ctx, int B, int nt, double* E, size_t strideE, cudaStream_t s)
{
    identity_rows<<<dim3(ntiles_lower(nt), B), kThreads, 0, s>>>(E, strideE);
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

static size_t const_smem(int lmax) { return sizeof(double) * 4 * (size_t)(lmax + 1); }

int fp64_build_tiled_into(cg_ctx* ctx, int B, const double* d_cl, bool add_noise, double* A, cudaStream_t s)
{
    const int ntile = ntiles_lower(ctx->nt);
    build_c_ref<<<dim3(ntile, B), kThreads, const_smem(ctx->lmax), s>>>(
        ctx->n, ctx->N, ctx->lmax, ctx->d_xyz, ctx->d_noise, ctx->d_lega, ctx->d_legb, ctx->d_beam, d_cl,
        add_noise ? 1 : 0, A, tiled_elems(ctx->nt));
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_build_packed(cg_ctx* ctx, int B, const double* d_cl, double* d_out, cudaStream_t s)
{
    const long np = (long)ctx->n * (ctx->n + 1) / 2;
    const unsigned gx = (unsigned)((np + kPairs * kThreads - 1) / (kPairs * kThreads));
    const int L1 = ctx->lmax + 1;
    auto run = [&](auto kernel, int nb) {
        kernel<<<dim3(gx, (B + nb - 1) / nb), kThreads, (sizeof(PackedL) + nb * sizeof(PackedTerm)) * L1, s>>>(
            ctx->n, ctx->N, ctx->lmax, B, ctx->d_xyz, ctx->d_lega, ctx->d_legb, ctx->d_beam, d_cl, d_out);
    };
    if (B == 1) run(build_c_packed<1>, 1);
    else if (B == 2) run(build_c_packed<2>, 2);
    else run(build_c_packed<4>, 4);
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_build_fiducial(cg_ctx* ctx, int lo, int hi, const double* d_tab, double m0, double* d_out, cudaStream_t s)
{
    const long np = (long)ctx->n * (ctx->n + 1) / 2;
    const int smem = (int)(sizeof(double) * 4 * (hi + 1));
    if (smem > 48 * 1024)
        CG_CUDA_TRY(ctx, cudaFuncSetAttribute(build_fid_packed, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    build_fid_packed<<<(unsigned)((np + 4 * kThreads - 1) / (4 * kThreads)), kThreads, smem, s>>>(
        ctx->n, ctx->N, lo, hi, ctx->d_xyz, d_tab, m0, d_out);
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_pol_matrix(cg_ctx* ctx, int n, int ld, const double* d_c_packed, const double* d_ninv, double* d_cd,
                    double* d_t, double* d_m, double* d_m_packed, unsigned char* work, int* scale, int* err,
                    cudaStream_t s)
{
    const size_t nel = (size_t)ld * ld;
    const int nt = ld / TS;
    packed_to_dense<<<(unsigned)((nel + kThreads - 1) / kThreads), kThreads, 0, s>>>(n, ld, d_c_packed, d_cd);
    CG_CUDA_TRY(ctx, cudaMemsetAsync(d_t, 0, sizeof(double) * nel, s));
    dense_to_tiles<<<dim3(nt, nt), kThreads, 0, s>>>(ld, d_ninv, d_m);
    // C's scales: C in the units of its diagonal has entries of one size, and so has T = C N^-1; N^-1 keeps only what
    // its own correlations give it (a scale taken from N^-1 would instead spread C over the noise's range)
    int rc = digit_scales(ctx, ld, d_cd, scale, s);
    if (!rc) rc = digit_gemm(ctx, nt, d_cd, d_ninv, false, d_t, scale, 1, work, err, s);      // T = C N^-1
    if (!rc) rc = digit_gemm(ctx, nt, d_ninv, d_t, true, d_m, scale, -1, work, err, s);  // M = N^-1 + N^-1 T
    if (rc) return rc;
    const long np = (long)n * (n + 1) / 2;
    tiles_to_packed<<<(unsigned)((np + kThreads - 1) / kThreads), kThreads, 0, s>>>(n, nt, d_m, d_m_packed);
    count_launch(ctx, 3);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_dense_residual(cg_ctx* ctx, int n, int ld, const double* d_ninv, const double* d_v, const double* d_s,
                        double* d_w, cudaStream_t s)
{
    dense_residual<<<(n + 7) / 8, kThreads, 0, s>>>(n, ld, d_ninv, d_v, d_s, d_w);
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_legendre_table(cg_ctx* ctx, int l0, int l1, const double* d_a, const double* d_b, double* d_out,
                        cudaStream_t s)
{
    const long np = (long)ctx->n * (ctx->n + 1) / 2;
    legendre_table<<<(unsigned)((np + kThreads - 1) / kThreads), kThreads, 0, s>>>(ctx->n, ctx->N, l0, l1, ctx->d_xyz,
                                                                                 d_a, d_b, d_out);
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_noise_matrix(cg_ctx* ctx, int nsims, int n, const double* d_sims, double* d_out, double* d_mean,
                      cudaStream_t s)
{
    const long nt = (n + kNoiseT - 1) / kNoiseT;
    noise_syrk_packed<<<(unsigned)(nt * (nt + 1) / 2), kThreads, 0, s>>>(nsims, n, d_sims, d_out);
    sim_means<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(nsims, n, d_sims, d_mean);
    count_launch(ctx, 2);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int fp64_loglike(cg_ctx* ctx, int B, const double* d_cl, const double* d_d, int d_stride, double* d_m2lnl,
                 double* d_chi2, double* d_logdet, double* d_grad, int* d_status, cudaStream_t s)
{
    const bool grad = d_grad != nullptr;
    int rc = fp64_ensure(ctx, B);
    if (!rc && grad && ctx->harm) rc = fp64_harmonics(ctx, s);
    if (rc) return rc;
    Fp64Work& w = ctx->w64;
    const int nt = ctx->nt, N = ctx->N, n = ctx->n, lmax = ctx->lmax;
    const size_t strideA = tiled_elems(nt);
    const int ntile = ntiles_lower(nt), ne = ext_blocks(ctx, grad);
    const bool inverse = grad && !ctx->harm;
    stage_mark(ctx, ST_BUILD, s);
    // The small kernels on either side of the factorisation overlap each other's ends, and ext_rows runs beside the
    // build (one value at nside 4 318 -> 304 us, a gradient at nside 8 691 -> 671).
    legendre_weights<<<B, kThreads, 0, s>>>(lmax, ctx->d_beam, d_cl, w.wfix, w.wexp, w.st, w.err);
    count_launch(ctx);
    // one element per thread block below four: twice the blocks of the shared form, and a single
    // element has nothing to share
    const int nb = B >= 4 ? 4 : 1;
    if ((rc = launch(ctx, nb == 4 ? build_c_tiled<4> : build_c_tiled<1>, dim3(ntile * kBuildParts, (B + nb - 1) / nb), kThreads,
                     sizeof(Split64) * (nb + 1) * (lmax + 1), 1, s, n, N, lmax, B, ctx->d_xyz, ctx->d_noise, w.wfix,
                     w.wexp, w.A, strideA)))
        return rc;
    const int drow = grad ? nharm_of(lmax) : 0;
    if (inverse) {
        if ((rc = fp64_identity_rows(ctx, B, nt, w.E, w.ext_elems, s))) return rc;
    } else {
        if ((rc = launch(ctx, ext_rows, dim3(nt, ne, B), kThreads, 0, 1, s, n, nt, drow, grad ? w.Yt : nullptr, d_d, d_stride,
                         w.E, w.ext_elems)))
            return rc;
    }
    stage_mark(ctx, ST_CHOL, s);
    if ((rc = digit_factor(ctx, B, nt, ne, inverse ? DIGIT_EXT_IDENTITY : DIGIT_EXT_ROWS, w.A, strideA, w.E,
                           w.ext_elems, w.diag, w.st, w.dig, w.err, s)))
        return rc;
    stage_mark(ctx, ST_SOLVE, s);
    if ((rc = launch(ctx, logdet_reduce, dim3(B), kLogThreads, 0, 1, s, n, N, w.diag, w.st, w.err, w.ld))) return rc;
    if (inverse) {
        pad_data<<<dim3((N + 255) / 256, B), 256, 0, s>>>(n, N, B, d_d, d_stride, w.dvec);
        symv_tiled<double><<<dim3(nt, B), kThreads, 0, s>>>(nt, N, w.A, strideA, w.dvec, w.alpha);
        chi2_finish<<<B, kThreads, 0, s>>>(n, N, w.dvec, w.alpha, w.ld, w.st, w.err, d_m2lnl, d_chi2);
        count_launch(ctx, 3);
        if (d_logdet) CG_CUDA_TRY(ctx, cudaMemcpyAsync(d_logdet, w.ld, sizeof(double) * B, cudaMemcpyDeviceToDevice, s));
    } else if ((rc = launch(ctx, chi2_rows, dim3(B), kThreads, 0, 1, s, nt, drow, w.E, w.ext_elems, w.ld, w.st, w.err, w.alpha,
                            d_m2lnl, d_chi2, d_logdet))) {
        return rc;
    }
    stage_mark(ctx, ST_ADJOINT, s);
    if (inverse) {
        for (int l0 = 2; l0 <= lmax; l0 += kAdjChunk) {
            const int l1 = (l0 + kAdjChunk <= lmax + 1) ? l0 + kAdjChunk : lmax + 1;
            adjoint_tiles<<<dim3(ntile, B), kThreads, 0, s>>>(n, N, l0, l1, ctx->d_xyz, ctx->d_lega, ctx->d_legb, w.A,
                                                              strideA, w.alpha, w.gpart, ntile, lmax + 1);
            count_launch(ctx);
        }
        adjoint_finish<<<B, 64, 0, s>>>(lmax, ntile, w.gpart, ctx->d_beam, w.st, w.err, d_grad);
        count_launch(ctx);
    } else if (grad) {
        if ((rc = launch(ctx, harmonic_sums, dim3(ne, kHarmSplit, B), kThreads, 0, 1, s, nt, ne, w.E, w.ext_elems, w.alpha,
                         w.gpart)) ||
            (rc = launch(ctx, harmonic_grad, dim3((lmax + 8) / 8, B), kThreads, 0, 1, s, lmax, ne, w.gpart, w.st, w.err,
                         d_grad)))
            return rc;
    }
    if (d_status && (rc = launch(ctx, copy_status, dim3((B + 127) / 128), 128, 0, 1, s, B, w.st, w.err, d_status))) return rc;
    stage_mark(ctx, ST_END, s);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

}  // namespace cg
