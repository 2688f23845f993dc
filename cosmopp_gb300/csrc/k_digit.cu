// FP64 Cholesky, triangular solve and inverse on the tensor cores.
//
// The FP64 pipe of this GPU gives 1.2 TFLOP/s, about 2 FMAs per cycle and SM, and a factorisation
// on it (k_chol.cu) runs at 83 % of that: the arithmetic is the bound.  Here every O(n^3) product is
// formed from exact BF16 products instead, by error-free splitting of the operands (Ozaki, Ogita,
// Oishi and Rump 2012; on tensor cores Mukunoki, Ozaki, Ogita and Imamura 2020):
//
//   * each row of an operand block (64 columns) gets a power of two 2^e above its largest entry and
//     is rounded to a 55-bit fixed-point number x = 2^(e-54) X, X written in seven signed base-256
//     digits d_0 .. d_6 (|d| <= 128), each exact in BF16;
//   * the digit products i + j <= 7 run on the tensor cores, summed over the 64 columns in eight FP32
//     accumulators, one per i + j.  Every partial sum is a whole number below 2^23 (64 columns, at
//     most 6 pairs of 2^14), so FP32 accumulation is exact;
//   * the eight sums are joined in 64-bit integers, rounded once at 2^-55 of the rows' scales, and
//     subtracted from the FP64 matrix: one FP64 rounding per 64 columns where an FMA chain has 64.
//
// The factorisation is right-looking on the trapezoid [A; E]: A the covariance in lower 64 x 64 tiles,
// E extra rows below it, which end as E L^-T.  With E = [harmonics; map]^T this is the whole
// likelihood: y = L^-1 d, Z = L^-1 Y.  With E = identity it is M^T, M = L^-1, and the same update
// kernel also sums V = M^T M = A^-1.  Per step k (64 columns):
//
//   digit_diag    L_kk and its inverse (FP64, one CTA per matrix), the inverse in digits
//   digit_panel   L_ik = S_ik L_kk^-T for the rows below and E's rows, left in digits
//   digit_update  S_ij -= L_ik L_jk^T over the trailing trapezoid, V_ij += M_ki^T M_kj
//
// Rows are kept in pairs of 64-row blocks; a pair's digits of the current column form one image,
// [8 k-cores][7 digits][8 row groups][2 blocks][8 rows][16 bytes], which serves as the A operand (128
// rows: groups 128 bytes apart) and, one block at a time, as the B operand (64 rows of four digits as
// N = 256: groups 256 bytes apart).
//
// A row with an infinity or a NaN gets the exponent kNonFinite, which makes everything it enters NaN.
#include <algorithm>

#include "cg_internal.h"
#include "cg_tc.cuh"

namespace cg {

namespace {

using namespace tc;

constexpr int kDig = 7;                     // digits per number
constexpr int kGroupBytes = 128;            // 8 rows x 16 bytes
constexpr int kPlane = 16 * kGroupBytes;    // one digit of 128 rows, 8 columns
constexpr int kCore = kDig * kPlane;        // 8 columns of a pair image
constexpr int kImg = 8 * kCore;             // a pair image: 114688 bytes
constexpr int kDPlane = 8 * kGroupBytes;    // the same for the 64 rows of an inverted diagonal block
constexpr int kDCore = kDig * kDPlane;
constexpr int kDImg = 8 * kDCore;           // 57344 bytes
constexpr int kNonFinite = 1 << 20;
constexpr int kThreads = 256;
constexpr uint32_t kWaits = 1u << 24;

// M64 N: bf16 x bf16 -> fp32, both operands K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// the digit products of 16 columns (k-cores 2 kc, 2 kc + 1): digit i of A against runs of digits of B,
// which land in consecutive 64-column accumulators i + j; the first column chunk initialises them
__device__ __forceinline__ void issue_products(uint32_t tmem, uint64_t a, uint64_t b, uint32_t a_plane,
                                               uint32_t b_plane, bool first)
{
    const uint32_t acc = first ? 0u : 1u;
    auto run = [&](int i, int j, int cnt, uint32_t ac) {
        mma_bf16(tmem + 64 * (i + j), a + (uint64_t)i * (a_plane >> 4), b + (uint64_t)j * (b_plane >> 4),
                 idesc_bf16(128, 64 * cnt), ac);
    };
    run(0, 0, 4, acc);
    run(0, 4, 3, acc);
    run(1, 6, 1, acc);  // accumulator 7 starts here
    run(1, 0, 4, 1);
    run(1, 4, 2, 1);
    run(2, 0, 4, 1);
    run(2, 4, 2, 1);
    run(3, 0, 4, 1);
    run(3, 4, 1, 1);
    run(4, 0, 4, 1);
    run(5, 0, 3, 1);
    run(6, 0, 2, 1);
}

// eight columns of all eight accumulators (64 columns apart), load and wait in one statement
__device__ __forceinline__ void tmem_ld_acc(uint32_t t, uint32_t (&r)[8][8])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%65];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%66];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%67];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%32, %33, %34, %35, %36, %37, %38, %39}, [%68];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%40, %41, %42, %43, %44, %45, %46, %47}, [%69];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%48, %49, %50, %51, %52, %53, %54, %55}, [%70];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%56, %57, %58, %59, %60, %61, %62, %63}, [%71];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[0][4]), "=r"(r[0][5]), "=r"(r[0][6]),
          "=r"(r[0][7]), "=r"(r[1][0]), "=r"(r[1][1]), "=r"(r[1][2]), "=r"(r[1][3]), "=r"(r[1][4]), "=r"(r[1][5]),
          "=r"(r[1][6]), "=r"(r[1][7]), "=r"(r[2][0]), "=r"(r[2][1]), "=r"(r[2][2]), "=r"(r[2][3]), "=r"(r[2][4]),
          "=r"(r[2][5]), "=r"(r[2][6]), "=r"(r[2][7]), "=r"(r[3][0]), "=r"(r[3][1]), "=r"(r[3][2]), "=r"(r[3][3]),
          "=r"(r[3][4]), "=r"(r[3][5]), "=r"(r[3][6]), "=r"(r[3][7]), "=r"(r[4][0]), "=r"(r[4][1]), "=r"(r[4][2]),
          "=r"(r[4][3]), "=r"(r[4][4]), "=r"(r[4][5]), "=r"(r[4][6]), "=r"(r[4][7]), "=r"(r[5][0]), "=r"(r[5][1]),
          "=r"(r[5][2]), "=r"(r[5][3]), "=r"(r[5][4]), "=r"(r[5][5]), "=r"(r[5][6]), "=r"(r[5][7]), "=r"(r[6][0]),
          "=r"(r[6][1]), "=r"(r[6][2]), "=r"(r[6][3]), "=r"(r[6][4]), "=r"(r[6][5]), "=r"(r[6][6]), "=r"(r[6][7]),
          "=r"(r[7][0]), "=r"(r[7][1]), "=r"(r[7][2]), "=r"(r[7][3]), "=r"(r[7][4]), "=r"(r[7][5]), "=r"(r[7][6]),
          "=r"(r[7][7])
        : "r"(t), "r"(t + 64), "r"(t + 128), "r"(t + 192), "r"(t + 256), "r"(t + 320), "r"(t + 384), "r"(t + 448)
        : "memory");
}

// the eight accumulators of one entry joined: units of 2^(ea + eb - 55), rounded to the nearest
__device__ __forceinline__ long long join_acc(const uint32_t (&r)[8][8], int q)
{
    auto v = [&](int s) { return (long long)__float2int_rn(__uint_as_float(r[s][q])); };
    const long long hi = v(0) * 16777216 + (v(1) * 65536 + (v(2) * 256 + v(3)));
    const long long lo = v(4) * 16777216 + (v(5) * 65536 + (v(6) * 256 + (v(7) + 4096)));
    return (hi << 19) + (lo >> 13);
}

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
// the row's exponent from the largest exponent field of its entries: |v| < 2^e
__device__ __forceinline__ int row_exp(int field) { return field == 0x7ff ? kNonFinite : field - 1022; }

// v as 2^(e-54) X, |v| < 2^e, X rounded to the nearest
__device__ __forceinline__ long long to_fixed(double v, int e)
{
    const long long bits = __double_as_longlong(v);
    const int f = (int)((unsigned long long)bits >> 52) & 0x7ff;
    unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
    int r = e - (f - 1075) - 53;
    if (f == 0 || r > 56) return 0;
    if (r < 0) r = 0;  // only with a non-finite entry, whose row is marked
    const long long x = (long long)(((m << 2 >> r) + 1) >> 1);
    return bits < 0 ? -x : x;
}

// X as two's complement digits, byte p the digit of weight 256^p (bytes 0 .. 5 balanced, byte 6 the top)
__device__ __forceinline__ unsigned long long to_digits(long long x)
{
    return ((unsigned long long)x + 0x0000808080808080ull) ^ 0x0000808080808080ull;
}

// byte p of two digit strings as a BF16 pair: with d = m - 128 s (m seven bits, s the sign bit),
// 128 + m and 128 + 128 s are BF16 numbers of the same exponent range, and their difference is exact
__device__ __forceinline__ uint32_t digit_pair(unsigned long long a, unsigned long long b, int p)
{
    const uint32_t wa = p < 4 ? (uint32_t)a : (uint32_t)(a >> 32), wb = p < 4 ? (uint32_t)b : (uint32_t)(b >> 32);
    const uint32_t q = p & 3;
    const uint32_t w = __byte_perm(wa, wb, q | (q << 4) | ((4 + q) << 8) | ((4 + q) << 12));
    const uint32_t m = (w & 0x007f007fu) | 0x43004300u, s = (w & 0x00800080u) | 0x43004300u;
    uint32_t d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(m), "r"(s));
    return d;
}

// eight numbers of one row: 16 bytes per digit, stored plane bytes apart (digit 0 = the top byte)
template <typename Store>
__device__ __forceinline__ void store_digits(const unsigned long long (&w)[8], Store&& store)
{
#pragma unroll
    for (int i = 0; i < kDig; ++i) {
        const int p = kDig - 1 - i;
        store(i, make_uint4(digit_pair(w[0], w[1], p), digit_pair(w[2], w[3], p), digit_pair(w[4], w[5], p),
                            digit_pair(w[6], w[7], p)));
    }
}

struct Dig {
    int nt, ne, ext;          // block rows of A and of E (both even); ext: DigitExt
    double* A;                // [B][strideA]
    double* E;                // [B][strideE]
    size_t strideA, strideE;  // doubles
    unsigned char* img;       // [B][pairs][kImg]
    int* ex;                  // [B][pairs][128]
    unsigned char* dimg;      // [B][kDImg]
    int* dex;                 // [B][64]
    int* err;
};

__device__ __forceinline__ int dig_pairs(const Dig& g) { return (g.nt + g.ne) / 2; }

// tile of E's block row eb at block column k
__device__ __forceinline__ double* ext_tile(const Dig& g, int b, int eb, int k)
{
    const size_t t = g.ext == DIGIT_EXT_IDENTITY ? (size_t)tile_index(k, eb) : (size_t)eb * g.nt + k;
    return g.E + (size_t)b * g.strideE + t * TILE_ELEMS;
}

// L_kk and its inverse in one sweep.  Thread (tr, tc) holds rows tr + 16 a, columns tc + 16 b.  At
// column c the trailing part is updated by the outer product of L's column c and the inverse's rows
// below c by that column times the inverse's finished row c, so the whole lower triangle takes part in
// every step and no second pass is needed.  All updates of an entry are summed apart (u) and
// subtracted once, when its column is reached.  87 k FMAs at 2 per cycle are half of the kernel's
// time; the rest is the chain of 64 pivots.
__global__ void __launch_bounds__(kThreads) digit_diag(int k, Dig g, double* __restrict__ diag,
                                                       int* __restrict__ status)
{
    __shared__ double colv[TS], rowv[TS], lv[TS], gv[TS];
    __shared__ double sx[TS][TS + 1];
    __shared__ int smax[4][TS];
    const int b = blockIdx.x, t = threadIdx.x, tr = t % 16, tc = t / 16;
    const double* tile = g.A + (size_t)b * g.strideA + (size_t)tile_index(k, k) * TILE_ELEMS;
    double s[4][4], u[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s[a][q] = q <= a ? tile[tr + 16 * a + TS * (tc + 16 * q)] : 0.0;
            u[a][q] = 0.0;
        }
    bool bad = false;
#pragma unroll
    for (int c1 = 0; c1 < 4; ++c1)
        for (int c0 = 0; c0 < 16; ++c0) {
            const int c = 16 * c1 + c0;
            if (tc == c0) {
#pragma unroll
                for (int a = c1; a < 4; ++a) colv[tr + 16 * a] = s[a][c1] - u[a][c1];
            }
            if (tr == c0) {
#pragma unroll
                for (int q = 0; q <= c1; ++q) rowv[tc + 16 * q] = -u[c1][q];
            }
            __syncthreads();
            if (t < 32) {
                double v = colv[c];
                if (!(v > 0.0)) {  // not positive definite (or NaN): flag, keep going on a benign value
                    bad = true;
                    v = 1.0;
                }
                const double inv = rsqrt(v);
                if (t == 0) diag[(size_t)b * g.nt * TS + k * TS + c] = v * inv;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = t + 32 * h;
                    const double l = (r > c ? colv[r] : rowv[r]) * inv;
                    const double x = r == c ? inv : l;
                    lv[r] = l;
                    gv[r] = x;
                    sx[c][r] = r <= c ? x : 0.0;
                }
            }
            __syncthreads();
#pragma unroll
            for (int a = c1; a < 4; ++a) {
                const int r = tr + 16 * a;
                const double l = r > c ? lv[r] : 0.0;
#pragma unroll
                for (int q = 0; q <= a; ++q) {
                    const int col = tc + 16 * q;
                    u[a][q] = fma(l, gv[col], col == c && r > c ? 0.0 : u[a][q]);
                }
            }
        }
    __syncthreads();
    if (t == 0 && bad && status[b] == CG_OK) status[b] = CG_ERR_NOT_PD;
    // the inverse's rows in digits: thread (row r, columns 16 q .. 16 q + 15)
    const int r = t % TS, q = t / TS;
    int f = 0;
#pragma unroll
    for (int c = 0; c < 16; ++c) f = max(f, exp_field(sx[r][16 * q + c]));
    smax[q][r] = f;
    __syncthreads();
    const int e = row_exp(max(max(smax[0][r], smax[1][r]), max(smax[2][r], smax[3][r])));
    if (q == 0) g.dex[(size_t)b * TS + r] = e;
    unsigned char* out = g.dimg + (size_t)b * kDImg;
#pragma unroll
    for (int kc = 0; kc < 2; ++kc) {
        unsigned long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] = to_digits(to_fixed(sx[r][16 * q + 8 * kc + c], e));
        unsigned char* o = out + (2 * q + kc) * kDCore + r * 16;
        store_digits(w, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(o + i * kDPlane) = v; });
    }
}

// Panel of step k, one CTA per row pair: rows x (64 columns) times the inverted diagonal block, the
// products formed as above, the result rounded row by row to digits without passing through FP64
// (E's rows also to FP64, which the solve and the gradient read).
constexpr int kPanelA = 0, kPanelB = kImg, kPanelTail = kImg + kDImg;
constexpr int kPanelSmem = kPanelTail + 2 * 128 * 4 + TS * 4 + 64;

__global__ void __launch_bounds__(kThreads, 1) digit_panel(int k, Dig g)
{
    extern __shared__ __align__(128) unsigned char sm[];
    int* smax = reinterpret_cast<int*>(sm + kPanelTail);  // [2][128]
    int* deb = smax + 256;                                // [64]
    __shared__ uint64_t full, done;
    __shared__ uint32_t tptr;
    const int t = threadIdx.x, b = blockIdx.y, m = t & 127, ch = t >> 7, warp = t >> 5;
    const int q0 = (k + 1) / 2, nq = g.nt / 2 - q0;
    const bool isext = (int)blockIdx.x >= nq;
    const int pair = isext ? g.nt / 2 + (int)blockIdx.x - nq : q0 + (int)blockIdx.x;
    const int half = (m >> 3) & 1, r = (m >> 4) * 8 + (m & 7);
    const int blk = 2 * pair + half, eb = blk - g.nt;
    const bool valid = isext ? (g.ext != DIGIT_EXT_IDENTITY || eb <= k) : blk > k;
    if (warp == 0) tmem_alloc(&tptr, 512);
    if (t == 0) {
        mbar_init(&full, 1);
        mbar_init(&done, 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(&full, kDImg);
        bulk_g2s(smem_u32(sm + kPanelB), g.dimg + (size_t)b * kDImg, kDImg, &full);
    }
    if (t < TS) deb[t] = g.dex[(size_t)b * TS + t];
    double* tile = nullptr;
    double v[32];
    int f = 0;
    if (valid) {
        tile = isext ? ext_tile(g, b, eb, k)
                     : g.A + (size_t)b * g.strideA + (size_t)tile_index(blk, k) * TILE_ELEMS;
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = tile[r + TS * (32 * ch + c)];
#pragma unroll
        for (int c = 0; c < 32; ++c) f = max(f, exp_field(v[c]));
    } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = 0.0;
    }
    smax[128 * ch + m] = f;
    __syncthreads();
    const int ea = row_exp(max(smax[m], smax[128 + m]));
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
        unsigned long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] = to_digits(to_fixed(v[8 * kc + c], ea));
        unsigned char* o = sm + kPanelA + (4 * ch + kc) * kCore + m * 16;
        store_digits(w, [&](int i, uint4 d) { *reinterpret_cast<uint4*>(o + i * kPlane) = d; });
    }
    fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tptr;
    bool ok = true;
    if (t == 0) {
        ok = mbar_wait(&full, 0, kWaits, g.err);
        const uint64_t ad = smem_desc(smem_u32(sm + kPanelA), kCore, kGroupBytes);
        const uint64_t bd = smem_desc(smem_u32(sm + kPanelB), kDCore, kGroupBytes);
        for (int kc = 0; kc < 4; ++kc)
            issue_products(tmem, ad + (uint64_t)kc * (2 * kCore >> 4), bd + (uint64_t)kc * (2 * kDCore >> 4), kPlane,
                           kDPlane, kc == 0);
        mma_commit(&done);
    }
    __syncwarp();
    ok = mbar_wait(&done, 0, kWaits, g.err) && ok;
    if (!ok) atomicExch(g.err, 1);
    fence_after();
    __syncwarp();
    // this thread's row, columns 32 ch .. 32 ch + 31, in units of 2^(ea + deb[c] - 55)
    long long u[32];
    int top = -(1 << 28);
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
        uint32_t acc[8][8];
        tmem_ld_acc(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 32 * ch + 8 * c8, acc);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const long long x = join_acc(acc, c);
            u[8 * c8 + c] = x;
            const int e = deb[32 * ch + 8 * c8 + c];
            if (x != 0 || e == kNonFinite) top = max(top, e + 64 - __clzll(x < 0 ? -x : x));
        }
    }
    fence_before();
    __syncthreads();  // smax is free again (its readers passed the barrier above the products)
    if (warp == 0) tmem_dealloc(tmem, 512);
    smax[128 * ch + m] = top;
    __syncthreads();
    top = max(smax[m], smax[128 + m]);
    const bool nonfinite = ea == kNonFinite || top > kNonFinite / 2;
    const int e = nonfinite ? kNonFinite : top < -(1 << 27) ? -1022 : top + ea - 55;
    if (!valid) return;
    if (ch == 0) g.ex[((size_t)b * dig_pairs(g) + pair) * 128 + 64 * half + r] = e;
    unsigned char* out = g.img + ((size_t)b * dig_pairs(g) + pair) * kImg + (size_t)m * 16;
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
        unsigned long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            // X = u 2^(deb - top + 54): |u| < 2^(top - deb), so |X| < 2^54
            const int sh = deb[32 * ch + 8 * kc + c] - top + 54;
            const long long x = u[8 * kc + c];
            long long y = 0;
            if (!nonfinite) {
                if (sh >= 0) y = x << min(sh, 63);
                else if (sh > -64) y = ((x >> (-sh - 1)) + 1) >> 1;
            }
            w[c] = to_digits(y);
        }
        unsigned char* o = out + (4 * ch + kc) * kCore;
        store_digits(w, [&](int i, uint4 d) { *reinterpret_cast<uint4*>(o + i * kPlane) = d; });
    }
    if (isext && g.ext == DIGIT_EXT_ROWS) {
#pragma unroll
        for (int c = 0; c < 32; ++c)
            tile[r + TS * (32 * ch + c)] = scaled(u[c], ea + deb[32 * ch + c] - 55);
    }
}

// Update of step k: persistent CTAs over (pair, pair) jobs of 128 x 128 outputs, K = 64.  Both images
// (2 x 112 KB) fill the shared memory; the 64 columns of each half of the second pair are one pass, with
// eight FP32 accumulators of 64 columns: all 512 tensor-memory columns.  The next job's images are
// fetched while the last pass is joined and subtracted.
constexpr int kUpB = kImg, kUpTail = 2 * kImg;
constexpr int kUpSmem = kUpTail + 2 * 128 * 4;

struct UpJob {
    int b, kind, p, q;        // kind 0: A's trailing part, 1: E's rows, 2: V = M^T M; q: columns, p: rows
    int pa, pb;               // images
};

__device__ __forceinline__ UpJob up_job(const Dig& g, int k, int per, int npe, int job)
{
    UpJob j;
    j.b = job / per;
    int l = job % per;
    const int nq = g.nt / 2, q0 = (k + 1) / 2, m = nq - q0, tri = m * (m + 1) / 2;
    if (l < tri) {
        int I, J;
        tile_coords(tri - 1 - l, I, J);  // columns in order, the next diagonal block's first
        j.kind = 0;
        j.q = nq - 1 - I;
        j.p = nq - 1 - J;
        j.pa = j.p;
        j.pb = j.q;
        return j;
    }
    l -= tri;
    if (l < npe * m) {
        j.kind = 1;
        j.q = q0 + l / npe;
        j.p = l % npe;
        j.pa = nq + j.p;
        j.pb = j.q;
        return j;
    }
    l -= npe * m;
    tile_coords(l, j.p, j.q);
    j.kind = 2;
    j.pa = nq + j.p;
    j.pb = nq + j.q;
    return j;
}

__global__ void __launch_bounds__(kThreads, 1) digit_update(int k, int njobs, int per, int npe, Dig g)
{
    extern __shared__ __align__(128) unsigned char sm[];
    int* sex = reinterpret_cast<int*>(sm + kUpTail);  // [2][128] exponents of the column pair
    __shared__ uint64_t full[4], done;
    __shared__ uint32_t tptr;
    const int t = threadIdx.x, warp = t >> 5, m = t & 127, ch = t >> 7;
    const int half = (m >> 3) & 1, r = (m >> 4) * 8 + (m & 7);
    const int pairs = dig_pairs(g);
    if (warp == 0) tmem_alloc(&tptr, 512);
    auto fetch = [&](const UpJob& j) {  // thread 0: both images, 16 columns per barrier
        const unsigned char* a = g.img + ((size_t)j.b * pairs + j.pa) * kImg;
        const unsigned char* bb = g.img + ((size_t)j.b * pairs + j.pb) * kImg;
        for (int kc = 0; kc < 4; ++kc) {
            mbar_arrive_expect_tx(&full[kc], (j.pa == j.pb ? 2 : 4) * kCore);
            bulk_g2s(smem_u32(sm + 2 * kc * kCore), a + 2 * kc * kCore, 2 * kCore, &full[kc]);
            if (j.pa != j.pb)
                bulk_g2s(smem_u32(sm + kUpB + 2 * kc * kCore), bb + 2 * kc * kCore, 2 * kCore, &full[kc]);
        }
    };
    int job = blockIdx.x;
    UpJob j = up_job(g, k, per, npe, job);
    if (t == 0) {
        for (int kc = 0; kc < 4; ++kc) mbar_init(&full[kc], 1);
        mbar_init(&done, 1);
        fence_mbar_init();
        fetch(j);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tptr;
    uint32_t passes = 0, round = 0;
    bool ok = true;
    for (; job < njobs; job += gridDim.x, ++round) {
        // the half of the column pair that holds column k is not part of the update
        const int h0 = (j.kind != 2 && 2 * j.q <= k) ? 1 : 0;
        const int h1 = (j.kind == 2 && 2 * j.q + 1 > k) ? 1 : 2;
        int* se = sex + 128 * (round & 1);
        if (t < 128) se[t] = g.ex[((size_t)j.b * pairs + j.pb) * 128 + t];
        const int ea = g.ex[((size_t)j.b * pairs + j.pa) * 128 + 64 * half + r];
        const UpJob cur = j;
        for (int h = h0; h < h1; ++h) {
            if (t == 0) {
                const uint64_t ad = smem_desc(smem_u32(sm), kCore, kGroupBytes);
                const uint64_t bd = smem_desc(smem_u32(sm + (cur.pa == cur.pb ? 0 : kUpB) + h * kGroupBytes), kCore,
                                              2 * kGroupBytes);
                for (int kc = 0; kc < 4; ++kc) {
                    if (h == h0) ok = mbar_wait(&full[kc], round & 1, kWaits, g.err) && ok;
                    issue_products(tmem, ad + (uint64_t)kc * (2 * kCore >> 4), bd + (uint64_t)kc * (2 * kCore >> 4),
                                   kPlane, kPlane, kc == 0);
                }
                mma_commit(&done);
            }
            // where this row of the pass goes
            const int rb = 2 * cur.p + half, cb = 2 * cur.q + h;
            bool valid;
            double* tile;
            double* Ab = g.A + (size_t)cur.b * g.strideA;
            if (cur.kind == 0) {
                valid = rb > k && rb >= cb;
                tile = Ab + (size_t)(valid ? tile_index(rb, cb) : 0) * TILE_ELEMS;
            } else if (cur.kind == 1) {
                valid = g.ext != DIGIT_EXT_IDENTITY || rb <= k;
                tile = valid ? ext_tile(g, cur.b, rb, cb) : Ab;
            } else {
                valid = rb <= k && rb >= cb;
                tile = Ab + (size_t)(valid ? tile_index(rb, cb) : 0) * TILE_ELEMS;
            }
            const bool fresh = cur.kind == 2 && rb == k;  // V's row k starts here
            const bool read = valid && !fresh;
            double* dst = tile + r + TS * 32 * ch;
            double old[8], nxt[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) old[c] = read ? dst[TS * c] : 0.0;
            __syncwarp();
            ok = mbar_wait(&done, passes & 1, kWaits, g.err) && ok;
            ++passes;
            fence_after();
            if (t == 0 && h == h1 - 1 && job + (int)gridDim.x < njobs) {
                j = up_job(g, k, per, npe, job + gridDim.x);
                fetch(j);
            }
            __syncthreads();  // the column exponents are in place
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
                if (c8 < 3) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) nxt[c] = read ? dst[TS * (8 * (c8 + 1) + c)] : 0.0;
                }
                uint32_t acc[8][8];
                tmem_ld_acc(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 32 * ch + 8 * c8, acc);
                if (valid) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const double x = scaled(join_acc(acc, c), ea + se[64 * h + 32 * ch + 8 * c8 + c] - 55);
                        dst[TS * (8 * c8 + c)] = cur.kind == 2 ? old[c] + x : old[c] - x;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 8; ++c) old[c] = nxt[c];
            }
            fence_before();
            __syncthreads();
            fence_after();
        }
        if (job + (int)gridDim.x < njobs) j = up_job(g, k, per, npe, job + gridDim.x);
    }
    if (!ok) atomicExch(g.err, 1);
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace

size_t digit_bytes(int nt, int ne)
{
    const size_t pairs = (size_t)(nt + ne) / 2;
    return pairs * kImg + pairs * 128 * sizeof(int) + kDImg + TS * sizeof(int);
}

int digit_factor(cg_ctx* ctx, int B, int nt, int ne, int ext, double* A, size_t strideA, double* E,
                 size_t strideE, double* diag, int* status, unsigned char* work, int* err, cudaStream_t s)
{
    const size_t pairs = (size_t)(nt + ne) / 2;
    Dig g;
    g.nt = nt;
    g.ne = ne;
    g.ext = ext;
    g.A = A;
    g.E = E;
    g.strideA = strideA;
    g.strideE = strideE;
    g.img = work;
    g.dimg = g.img + (size_t)B * pairs * kImg;
    g.ex = reinterpret_cast<int*>(g.dimg + (size_t)B * kDImg);
    g.dex = g.ex + (size_t)B * pairs * 128;
    g.err = err;
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmem));
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_update, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpSmem));
    for (int k = 0; k < nt; ++k) {
        digit_diag<<<B, kThreads, 0, s>>>(k, g, diag, status);
        const int nq = nt / 2 - (k + 1) / 2;
        const int npe = ext == DIGIT_EXT_IDENTITY ? k / 2 + 1 : ne / 2;
        if (nq + npe == 0) { count_launch(ctx, 1); continue; }
        digit_panel<<<dim3(nq + npe, B), kThreads, kPanelSmem, s>>>(k, g);
        const int per = nq * (nq + 1) / 2 + npe * nq + (ext == DIGIT_EXT_IDENTITY ? npe * (npe + 1) / 2 : 0);
        count_launch(ctx, per > 0 ? 3 : 2);
        if (per > 0)
            digit_update<<<(unsigned)std::min<long long>((long long)per * B, ctx->sm_count), kThreads, kUpSmem, s>>>(
                k, per * B, per, npe, g);
    }
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

}  // namespace cg
