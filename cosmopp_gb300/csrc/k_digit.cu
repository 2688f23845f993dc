// FP64 Cholesky, triangular solve and inverse on the tensor cores.
//
// The FP64 pipe of this GPU gives 1.2 TFLOP/s, about 2 FMAs per cycle and SM, and a factorisation
// on it (k_chol.cu) runs at 83 % of that: the arithmetic is the bound.  Here every O(n^3) product is
// formed from exact BF16 products instead, by error-free splitting of the operands (Ozaki, Ogita,
// Oishi and Rump 2012; on tensor cores Mukunoki, Ozaki, Ogita and Imamura 2020):
//
//   * each row of an operand block (64 columns) gets a power of two 2^e above its largest entry and
//     is rounded to a 55-bit fixed-point number x = 2^(e-54) X, X written in seven signed base-256
//     digits d_0 .. d_6 (|d| <= 128), each exact in BF16.  An entry far below its row's largest thus keeps
//     fewer bits than in FP64, so the columns of an operand are brought to one scale first where the other
//     operand has the opposite one: S_ik = L_ik L_kk^T by the diagonal block's scales (diag_scale), the
//     products of digit_gemm by those of digit_scales.  L's own columns need none: row i of L has norm sqrt(A_ii);
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
//   digit_diag    L_kk (fixed point) and its inverse (FP64), four CTAs per matrix, the inverse in digits
//   digit_panel   L_ik = S_ik L_kk^-T for the rows below and E's rows, left in digits
//   digit_update  S_ij -= L_ik L_jk^T over the trailing trapezoid, V_ij += M_ki^T M_kj
//
// Rows are kept in pairs of 64-row blocks; a pair's digits of the current column form one image,
// [8 k-cores][7 digits][16 row groups][8 rows][16 bytes], which is the A operand as it stands (128 rows) and,
// 32 rows at a time, taken out by a tensor copy as [8][7][4][8][16 bytes], the B operand (the 7 digits of 32
// rows as N = 224, groups 128 bytes apart).
//
// Every wait on a barrier is bounded.  One that gives up sets *err, which all waits watch; its thread and those that see
// the flag skip their later waits and take no more work (the update after the job in hand), and the copies and products in flight are waited for, bounded
// too, before their shared and tensor memory is given up.
//
// A row with an infinity or a NaN gets the exponent kNonFinite, which makes everything it enters NaN.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cg_fixed.cuh"
#include "cg_internal.h"
#include "cg_launch.cuh"
#include "cg_tc.cuh"

namespace cg {

namespace {

using namespace tc;

constexpr int kDig = 7;                     // digits per number
constexpr int kGroupBytes = 128;            // 8 rows x 16 bytes
constexpr int kPlane = 16 * kGroupBytes;    // one digit of 128 rows, 8 columns
constexpr int kCore = kDig * kPlane;        // 8 columns of a pair image
constexpr int kImg = 8 * kCore;             // a pair image: 114688 bytes
constexpr int kPieceRow = 4 * kGroupBytes;  // a digit of the 32 rows of a piece
constexpr int kPieceCore = kDig * kPieceRow;
constexpr int kPiece = 8 * kPieceCore;      // 28672 bytes
constexpr int kDPlane = 8 * kGroupBytes;    // the same for the 64 rows of an inverted diagonal block
constexpr int kDCore = kDig * kDPlane;
constexpr int kDImg = 8 * kDCore;           // 57344 bytes
constexpr uint32_t kWaits = 1u << 22;       // attempts before a wait gives up

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
// which land in consecutive accumulators i + j of NC columns; the first column chunk initialises them
template <int NC>
__device__ __forceinline__ void issue_products(uint32_t tmem, uint64_t a, uint64_t b, uint32_t a_plane,
                                               uint32_t b_plane, bool first)
{
    const uint32_t acc = first ? 0u : 1u;
    auto run = [&](int i, int j, int cnt, uint32_t ac) {
        mma_bf16(tmem + NC * (i + j), a + (uint64_t)i * (a_plane >> 4), b + (uint64_t)j * (b_plane >> 4),
                 idesc_bf16(128, NC * cnt), ac);
    };
    // N is at most 256: 4 digits of 64 columns, all 7 of 32.  Fewer, wider instructions matter: each reads
    // A's digit again (with 4 digits of 32 columns at a time the operand reads held the tensor pipe for 65 % of
    // the update, its arithmetic for 37 %).
    constexpr int most = 256 / NC < kDig ? 256 / NC : kDig;
    if (first) run(1, 6, 1, 0u);  // accumulator 7 starts here
#pragma unroll
    for (int i = 0; i < kDig; ++i) {
        const int n = i == 0 ? kDig : i == 1 && first ? kDig - 1 : kDig + 1 - i;
#pragma unroll
        for (int j = 0; j < kDig; j += most)
            if (j < n) run(i, j, n - j < most ? n - j : most, i == 0 ? acc : 1u);
    }
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
    int nk;                   // sets of images that an update takes one after the other (1 in a factorisation)
    size_t kimg, kex;         // their distances
    int im0, kim;             // img and kimg as numbers of images from the start of the tensor map
    int prefetch;             // the matrices exceed L2: an update fetches the next job's tiles ahead
    unsigned char* dimg;      // [B][kDImg]
    int* dex;                 // [B][64]
    int* err;
    uint32_t waits;           // the diagonal block's and the panel's limit: kWaits, or 0 in the self-test
};

// a wait that gives up, or finds that another has, sets the flag and clears ok; later ones are skipped
__device__ __forceinline__ void bounded_wait(bool& ok, uint64_t* bar, uint32_t parity, int* err, uint32_t waits)
{
    if (!ok) return;
    ok = mbar_wait(bar, parity, waits, err);
    if (!ok) *(volatile int*)err = 1;
}

__device__ __forceinline__ int dig_pairs(const Dig& g) { return (g.nt + g.ne) / 2; }

// tile of E's block row eb at block column k
__device__ __forceinline__ double* ext_tile(const Dig& g, int b, int eb, int k)
{
    const size_t t = g.ext == DIGIT_EXT_IDENTITY ? (size_t)tile_index(k, eb) : (size_t)eb * g.nt + k;
    return g.E + (size_t)b * g.strideE + t * TILE_ELEMS;
}

// e with S_rr < 2^(2 e) for an entry of the diagonal: row r of the factor is below 2^e, and column r of what the
// panel multiplies by the inverse is scaled by 2^-e.  (With one exponent for a row of S and no scales, pixels of
// sigma 1 and 1e9 side by side left chi2 with a relative error of 1e-9 where the FP64 factorisation has 1e-15.)
__device__ __forceinline__ int diag_scale(double s) { return (exp_field(s) - 1022 + 1) >> 1; }

// a row's exponent from the largest of its entries' scaled_field: |v 2^-e| < 2^(row exponent)
__device__ __forceinline__ int scaled_field(double v, int e)
{
    const int f = exp_field(v);
    return f == 0x7ff ? kNonFinite : f == 0 ? -(1 << 28) : f - e;
}
__device__ __forceinline__ int scaled_row_exp(int field)
{
    return field > kNonFinite / 2 ? kNonFinite : field < -(1 << 27) ? -1022 : field - 1022;
}

// ---- diagonal block: L_kk in 64-bit fixed point, its inverse in FP64, one cluster per matrix ----
//
// The FP64 pipe takes a warp instruction every 64 cycles and SM partition, whatever its active lanes
// (a lone rsqrt is 456 cycles), so the 64 dependent pivots and the 44 k FMAs of a 64 x 64 factorisation
// in FP64 took 83 us with the inverse; this takes 30 us, 23 of them the chain of pivots.  CTA 0 factors the block in
// integers instead: row r is scaled by 2^-e_r, 2^(2 e_r) above S_rr, so that |S| and |L| are at most 1, held as 2^58
// times their value.  A product sum is three 32 x 32 -> 64 multiply-adds (64 per cycle) on L = h 2^29 + l: h h'
// and h l' + l h', l l' (below 2^-56 of a product) left out; the sums cannot overflow, since rows of L
// have norm at most 1 (sum h h' <= 2^58, sum of the cross terms <= 2^61).  All updates of an entry are
// thus summed exactly but for the last bits and subtracted once, when its column is reached.
//
// Within CTA 0 one warp factors the 4 x 4 diagonal block of a panel of four columns (the chain of pivots), two warps
// follow it with the panel's 64 rows and add the panel's products to the next panel's columns, the four rows of its
// diagonal block first; sixteen warps add them to the columns after that meanwhile.  (With the owners' sums in the
// chain a panel took 3.5 k cycles; this 3.0 k, 2.1 k of them the four pivots.)  The other CTAs of the cluster form 16
// to 24 columns each of the inverse in FP64 as the factor's columns arrive in their shared memory, eight rows at a
// time: those eight by one warp per eight columns, then eight products for every row below.  (One row at a time
// took 400 to 1000 cycles a row, which even seven CTAs of eight columns could not hide.)
constexpr int kDiagOwners = 512, kBlockThread = kDiagOwners + TS, kDiagThreads = kBlockThread + 32;
constexpr int kDiagCtas = 4, kPanel = 4;
constexpr int kFrac = 58, kLow = 29;

struct DiagFactor {                     // CTA 0
    longlong2 acc[TS][TS];              // column by column: an entry less its updates' high parts, their low parts
    long long group[2][8][TS];          // eight columns of L
    int4 lsp[2][kPanel / 2][TS];        // a panel's columns of L, split (h, l), two columns side by side
    longlong2 piv[2][kPanel];           // a pivot's inverse root: (c, a << 32 | m) of InvSqrt
    long long pv[2][kPanel];            // the pivot
    int2 sb[2][kPanel][2 * kPanel];     // the diagonal block's columns of L, split (rows past its last are not used)
    long long next[kPanel][kPanel];     // the next diagonal block
};
struct DiagInverse {                    // the other CTAs
    long long lq[8][8][TS];             // L's columns as they arrive, 8 groups
    double ld[2][8][TS];                // the current group in FP64, two buffers
    double x[TS][25];                   // rows of this CTA's columns: sums, then the inverse (and one against conflicts)
    double inv[2][8];                   // 1 / L_cc of the current group
    int smax[kDiagCtas][TS];            // row exponents of each CTA's part (0: this one's)
};
struct DiagShared {
    union {
        DiagFactor f;
        DiagInverse v;
    };
    long long yq[TS];                   // 1 / L_cc as yq 2^(yk - 61)
    int yk[TS];
    int e[TS];                          // row scales
    uint64_t full[8];
    int bad;
};

// the CTA's shared-memory address p in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(const void* p, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t a, long long v)
{
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, int v)
{
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// what this thread has written or seen written is visible to the thread that sees the arrival
__device__ __forceinline__ void arrive_cluster(uint64_t* bar, int rank)
{
    asm volatile("fence.acq_rel.cluster;\n\tmbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                     mapa(bar, rank))
                 : "memory");
}
__device__ __forceinline__ void wait_cluster(bool& ok, uint64_t* bar, uint32_t parity, const Dig& g)
{
    if (!ok) return;
    const uint32_t a = smem_u32(bar);
    const volatile int* err = g.err;
    for (uint32_t it = 0; it < g.waits; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return;
        if ((it & 255) == 255 && *err) break;
    }
    ok = false;
    *(volatile int*)g.err = 1;
}

// v 2^(kFrac - e) rounded to the nearest; false where |v| >= 2^e or v is not finite
__device__ __forceinline__ bool to_scaled(double v, int e, long long& x)
{
    const long long bits = __double_as_longlong(v);
    const int f = (int)((unsigned long long)bits >> 52) & 0x7ff, r = e - (f - 1022);
    x = 0;
    if (f == 0 || r > 60) return true;
    if (r < 0 || f == 0x7ff) return false;
    const unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | 0x10000000000000ull;
    const long long y = (long long)(((m << (kFrac - 52) >> r) + 1) >> 1);
    x = bits < 0 ? -y : y;
    return true;
}

// 1 / sqrt(v) for v > 0 to about 2^-58: an FP32 estimate y0 = m 2^(a - 54), m of 24 bits (relative error
// below 2^-21), and y0 (1 + c), c 2^-58 = h / 2 + 3 h^2 / 8, h = 1 - v y0^2 (the series of (1 - h)^(-1/2))
struct InvSqrt {
    unsigned m;
    int a;
    long long c;
};
__device__ __forceinline__ InvSqrt inv_sqrt(long long v)
{
    // v 2^-sh below 2^31 with at least 24 bits, sh even
    const int sh = v >= (1ll << 52) ? 28 : 33 - ((__clzll(v) - 1) | 1);
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)(int)(sh >= 0 ? v >> sh : v << -sh)));
    const unsigned bits = __float_as_uint(f);
    InvSqrt y;
    y.m = (bits & 0x7fffffu) | 0x800000u;
    y.a = (int)(bits >> 23) - 127 - 23 + 54 - sh / 2;
    // v 2^(2 a) m^2 is near 2^108: h = 1 - that, 2^58 times
    const unsigned long long m2 = ((unsigned long long)y.m * y.m) << 14, n = (unsigned long long)v << (2 * y.a);
    const unsigned ah = (unsigned)(n >> 31), al = (unsigned)n & 0x7fffffffu;
    const unsigned bh = (unsigned)(m2 >> 31), bl = (unsigned)m2 & 0x7fffffffu;
    const long long h = (1ll << 58) - (long long)(((unsigned long long)ah * bh >> 2) +
                                                  (((unsigned long long)ah * bl + (unsigned long long)al * bh) >> 33));
    const int hs = (int)(h >> 16);              // below 2^22
    y.c = (h >> 1) + ((3 * (long long)hs * hs) >> 29);
    return y;
}

// An entry of L beyond 1, which no positive definite matrix has and its numbers have no place for (mul_inv_sqrt wraps
// from |x| 2^a = 2^63 on, the sums from |L| = 4 on): xh the high word of the column's entry x, lh of what mul_inv_sqrt
// made of it.  |x| < 2^(62 - a), or 2^32 for a = 31, where its numbers are right, and |L| < 1 + 2^-26.
__device__ __forceinline__ bool beyond_one(int xh, int lh, int a)
{
    return (xh ^ (xh >> 31)) >> max(30 - a, 0) != 0 || (lh ^ (lh >> 31)) > 1 << (kFrac - 32);
}

// x y 2^(kFrac / 2) for |x| <= 2^(kFrac / 2) sqrt(v): an entry of L from the column's entry x
__device__ __forceinline__ long long mul_inv_sqrt(long long x, const InvSqrt& y)
{
    const long long z = x << y.a;               // below 2^61
    const int w = (int)(y.m << 7);
    const long long l0 =
        (long long)(int)(z >> 32) * w + (long long)(((unsigned long long)(unsigned)z * (unsigned)w) >> 32);
    // + l0 c 2^-58, |c| < 2^38, in 29 + 29 and 22 + 16 bits
    const int lh = (int)(l0 >> 29), ll = (int)(l0 & 0x1fffffff), ch = (int)(y.c >> 16), cl = (int)(y.c & 0xffff);
    return l0 + (((long long)lh * ch >> 13) + (((long long)lh * cl + ((long long)ll * ch >> 13)) >> 29));
}

__device__ __forceinline__ int2 split_low(long long l)
{
    const int lo = (int)(((l + (1ll << (kLow - 1))) & ((1ll << kLow) - 1)) - (1ll << (kLow - 1)));
    return make_int2((int)((l - lo) >> kLow), lo);
}

// (a warp arrives once: its lanes are brought together first)
__device__ __forceinline__ void named_sync(int id, int threads)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads)
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// thread i < kDiagOwners: group g of L's columns and pivots into the shared memory of the other CTAs
__device__ __forceinline__ void diag_publish(DiagShared& sh, int g, int i)
{
#pragma unroll
    for (int rank = 1; rank < kDiagCtas; ++rank) {
        st_cluster(mapa(&sh.v.lq[g][0][0] + i, rank), (&sh.f.group[g & 1][0][0])[i]);
        if (i < 8) {
            st_cluster(mapa(&sh.yq[8 * g + i], rank), sh.yq[8 * g + i]);
            st_cluster(mapa(&sh.yk[8 * g + i], rank), sh.yk[8 * g + i]);
        }
    }
}

// Named barriers of CTA 0.  With the panel's parity: kFact (L's columns are in lsp and group, 1 / L_cc in yq, and the
// owners are done with the panel before: every thread; the block warp only arrives), kCol + 2 j (column j of the panel's diagonal block is in piv,
// pv, sb: the row warps and the block warp, which may be a panel ahead of one of them).  kBase: the next panel's
// diagonal block lacks this panel only (the owners' warp and the row warp that have it); kNext: it is complete, in
// next (that row warp and the block warp).
constexpr int kFact = 1, kNext = 3, kBase = 4, kCol = 5;
constexpr int kColThreads = TS + 32, kNextThreads = 64;

// x - s q for split numbers of kFrac fraction bits
__device__ __forceinline__ long long sub_product(long long x, int2 s, int2 q)
{
    return x - ((long long)s.x * q.x + (((long long)s.x * q.y + (long long)s.y * q.x) >> kLow));
}

__device__ __forceinline__ long long shfl(long long v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ int2 shfl(int2 v, int lane)
{
    return make_int2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

__device__ __forceinline__ long long joined(longlong2 a) { return a.x - (a.y >> kLow); }

// an entry less the products of its row and column over a panel
__device__ __forceinline__ longlong2 less_product(longlong2 o, int4 x0, int4 x1, int4 y0, int4 y1)
{
    long long h = (long long)x0.x * y0.x, l = (long long)x0.x * y0.y, k = (long long)x1.x * y1.y;
    l += (long long)x0.y * y0.x;
    k += (long long)x1.y * y1.x;
    h += (long long)x0.z * y0.z;
    l += (long long)x0.z * y0.w;
    k += (long long)x1.z * y1.w;
    l += (long long)x0.w * y0.z;
    k += (long long)x1.w * y1.z;
    h += (long long)x1.x * y1.x;
    h += (long long)x1.z * y1.z;
    return make_longlong2(o.x - h, o.y + (l + k));
}

// The owners' loop stays rolled: their sums in registers, 96 multiply-adds unrolled, ran at 8 cycles an instruction,
// which each warp fetched anew for every panel.

// The diagonal blocks of all panels, one warp, row lane % 4 each; panel p has columns 4 p .. 4 p + 3.  Returns whether
// a pivot was not positive.
__device__ __forceinline__ bool diag_blocks(DiagShared& sh)
{
    constexpr int np = TS / kPanel;
    DiagFactor& f = sh.f;
    const int lane = threadIdx.x & 31, q = lane & (kPanel - 1);
    bool bad = false;
    long long x[kPanel];  // the row's entries from the current column on
#pragma unroll
    for (int j = 0; j < kPanel; ++j) x[j] = f.acc[j][q].x;
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
        const int buf = p & 1;
        long long next = x[0];
#pragma unroll
        for (int j = 0; j < kPanel; ++j) {
            long long v = shfl(next, j);
            if (v <= 0) {  // not positive definite: flag, keep going on a benign value
                bad = true;
                v = 1ll << kFrac;
            }
            const InvSqrt y = inv_sqrt(v);
            const int2 s = split_low(mul_inv_sqrt(x[0], y));
            next = sub_product(x[1], s, s);  // in lane j + 1: the next pivot
            if (lane == 0) {
                f.piv[buf][j] = make_longlong2(y.c, ((long long)y.a << 32) | y.m);
                f.pv[buf][j] = v;
            }
            if (lane > j && lane < kPanel) f.sb[buf][j][lane] = s;
            named_arrive(kCol + 2 * j + buf, kColThreads);
#pragma unroll
            for (int i = 0; i + 1 < kPanel - j; ++i) x[i] = sub_product(x[i + 1], s, shfl(s, j + 1 + i));
        }
        __syncwarp();
        if (lane < kPanel) {  // 1 / L_cc
            const longlong2 w = f.piv[buf][lane];
            const long long m = (long long)(unsigned)w.y << 38;
            sh.yq[kPanel * p + lane] = m + (__mul64hi(m, w.x << 24) >> 18);
            sh.yk[kPanel * p + lane] = (int)(w.y >> 32) - 2;
        }
        named_arrive(kFact + buf, kDiagThreads);
        if (p + 1 < np) {
            named_sync(kNext, kNextThreads);
#pragma unroll
            for (int j = 0; j < kPanel; ++j) x[j] = f.next[q][j];
        }
    }
    return bad;
}

// The rows, row r per thread.  The owners' sums of a panel's columns lack the panel just before it, whose products the
// rows add themselves (of them the block warp gets the diagonal block): so the owners have a panel's time for theirs,
// and the chain of pivots passes through the rows only.  Returns whether an entry of L is beyond 1.
__device__ __forceinline__ bool diag_rows(DiagShared& sh, int r)
{
    constexpr int np = TS / kPanel;
    DiagFactor& f = sh.f;
    const int lane = r & 31, er = (lane >> 2) & 3, ec = lane & 3;
    bool beyond = false;
    long long x[kPanel];  // the row's entries from the current column on
#pragma unroll
    for (int j = 0; j < kPanel; ++j) x[j] = f.acc[j][r].x;
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
        const int buf = p & 1, c0 = kPanel * p, from = (c0 + kPanel) & 31;
        const bool completes = p + 1 < np && (c0 + kPanel) / 32 == r / 32;
        long long dh = 0, dl = 0;
        int xh[kPanel], lh[kPanel], ya[kPanel];
#pragma unroll
        for (int j = 0; j < kPanel; ++j) {
            named_sync(kCol + 2 * j + buf, kColThreads);
            const longlong2 w = f.piv[buf][j];
            InvSqrt y;
            y.c = w.x;
            y.m = (unsigned)w.y;
            y.a = (int)(w.y >> 32);
            if (r == c0 + j) x[0] = f.pv[buf][j];
            if (r < c0 + j) x[0] = 0;
            const long long l = mul_inv_sqrt(x[0], y);
            const int2 s = split_low(l);
            xh[j] = (int)(x[0] >> 32);
            lh[j] = (int)(l >> 32);
            ya[j] = y.a;
            const int2 a = shfl(s, from + er), b = shfl(s, from + ec);
            dh += (long long)a.x * b.x;
            dl += (long long)a.x * b.y;
            dl += (long long)a.y * b.x;
#pragma unroll
            for (int i = 0; i + 1 < kPanel; ++i) x[i] = sub_product(x[i + 1], s, f.sb[buf][j][j + 1 + i]);
            f.group[(p >> 1) & 1][(p & 1) * kPanel + j][r] = l;
            reinterpret_cast<int2*>(&f.lsp[buf][j / 2][r])[j & 1] = s;
        }
        if (completes) {
            if (p > 0) named_sync(kBase, kNextThreads);
            const longlong2 o = f.acc[c0 + kPanel + ec][c0 + kPanel + er];
            if (lane < 16) f.next[er][ec] = joined(make_longlong2(o.x - dh, o.y + dl));
            named_arrive(kNext, kNextThreads);
        }
        // (here, where the block warp does not wait for the rows)
#pragma unroll
        for (int j = 0; j < kPanel; ++j) beyond |= beyond_one(xh[j], lh[j], ya[j]);
        named_sync(kFact + buf, kDiagThreads);
        if (p + 1 == np) break;
        const int4 x0 = f.lsp[buf][0][r], x1 = f.lsp[buf][1][r];
#pragma unroll
        for (int j = 0; j < kPanel; ++j) {
            const int c = c0 + kPanel + j;
            x[j] = joined(less_product(f.acc[c][r], x0, x1, f.lsp[buf][0][c], f.lsp[buf][1][c]));
        }
    }
    return beyond;
}

__device__ __forceinline__ void diag_factor(DiagShared& sh, const double* __restrict__ tile)
{
    DiagFactor& f = sh.f;
    const int t = threadIdx.x;
    bool bad = false;
    for (int i = t; i < TILE_ELEMS; i += kDiagThreads) {
        const int r = i % TS, c = i / TS;
        long long x = 0;
        if (r >= c) bad |= !to_scaled(tile[i], sh.e[r] + sh.e[c], x);
        f.acc[c][r] = make_longlong2(x, 0);
    }
    if (bad) sh.bad = 1;
    __syncthreads();
    constexpr int np = TS / kPanel;
    if (t >= kDiagOwners) {
        if (t >= kBlockThread) {
            if (diag_blocks(sh) && t == kBlockThread) sh.bad = 1;
        } else {
            if (diag_rows(sh, t - kDiagOwners)) sh.bad = 1;
        }
    } else {
        // warp w has the columns of panel w: this thread column c, rows tr + 8 a
        const int w = t / 32, tr = t % 8, c = t / 8;
#pragma unroll 1
        for (int p = 0; p < np; ++p) {
            const int buf = p & 1;
            named_sync(kFact + buf, kDiagThreads);
            // the group published in the last step (every thread has passed its stores)
            if (p > 0 && (p & 1) == 0 && t < kDiagCtas - 1) arrive_cluster(&sh.full[p / 2 - 1], 1 + t);
            if (w > p + 1) {
                const int4 y0 = f.lsp[buf][0][c], y1 = f.lsp[buf][1][c];
#pragma unroll 2
                for (int r = tr + kPanel * (w & ~1); r < TS; r += 8)
                    f.acc[c][r] = less_product(f.acc[c][r], f.lsp[buf][0][r], f.lsp[buf][1][r], y0, y1);
                if (w == p + 2) named_arrive(kBase, kNextThreads);
            }
            if (p & 1) diag_publish(sh, p / 2, t);
        }
    }
    __syncthreads();
    if (t < kDiagCtas - 1) arrive_cluster(&sh.full[7], 1 + t);
}

// The blocks of eight columns of the inverse that CTA `rank` forms: block q takes (7 - q)(8 - q) / 2 products of 8 x 8,
// so 0, 6, 7 | 1, 4, 5 | 2, 3 (28, 30, 25 in all; in order, 0, 1 | 2, 3, 4 | 5, 6, 7, they were 49, 31, 4 and the first
// CTA ended 7 us after the factor).
__device__ __forceinline__ int diag_block_of(int rank, int j)
{
    return rank == 1 ? (j == 0 ? 0 : 5 + j) : rank == 2 ? (j == 0 ? 1 : 3 + j) : 2 + j;
}

// a cluster of kDiagCtas CTAs per matrix
__global__ void __launch_bounds__(kDiagThreads, 1)
    digit_diag(int k, Dig g, double* __restrict__ diag, int* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char sm[];
    DiagShared& sh = *reinterpret_cast<DiagShared*>(sm);
    const int rank = blockIdx.x % kDiagCtas, b = blockIdx.x / kDiagCtas, t = threadIdx.x;
    const double* tile = g.A + (size_t)b * g.strideA + (size_t)tile_index(k, k) * TILE_ELEMS;
    if (t < 8) mbar_init(&sh.full[t], 1);
    if (t == 0) sh.bad = 0;
    fence_mbar_init();
    wait_prior();
    launch_dependents();  // not before: the panel reads column k ahead of its own wait
    if (t < TS) sh.e[t] = diag_scale(tile[t * (TS + 1)]);
    cluster_barrier();
    if (rank == 0) {
        diag_factor(sh, tile);
        cluster_barrier();
        if (t == 0 && sh.bad && status[b] == CG_OK) status[b] = CG_ERR_NOT_PD;
        return;
    }
    if (t >= kDiagOwners) {  // the panel's warps: nothing to do here
        cluster_barrier();
        return;
    }
    DiagInverse& v = sh.v;
    const int nj = rank == 3 ? 2 : 3, first = rank - 1;
    auto block = [&](int j) { return diag_block_of(rank, j); };  // columns 8 block(j) .. 8 block(j) + 7
    if (t < TS) v.smax[0][t] = -(1 << 28);
    const int r = t / 8, qi = t % 8;
    double w[3] = {0.0, 0.0, 0.0};  // row r's sums, columns 8 block(j) + qi
    bool ok = true;
    for (int grp = 0; grp < 8; ++grp) {
        wait_cluster(ok, &sh.full[grp], 0, g);
        if (rank == 1 && t < 8) {  // L's diagonal
            const int c = 8 * grp + t;
            diag[(size_t)b * g.nt * TS + k * TS + c] = scaled(v.lq[grp][t][c], sh.e[c] - kFrac);
        }
        if (grp < first) continue;
        double (&ld)[8][TS] = v.ld[grp & 1];
        ld[t / TS][t % TS] = scaled(v.lq[grp][t / TS][t % TS], -kFrac);
        if (t < 8) v.inv[grp & 1][t] = scaled(sh.yq[8 * grp + t], sh.yk[8 * grp + t] - 61);
        // the group's eight rows: their sums to one warp per eight columns, which finishes them in order (lane:
        // rows u and u + 4, one column), then eight products for every row below
        if (r / 8 == grp) {
#pragma unroll
            for (int j = 0; j < 3; ++j)
                if (j < nj) v.x[r][qi + 8 * j] = w[j];
        }
        named_sync(1, kDiagOwners);
        if (t / 32 < nj) {
            const int u = (t % 32) / 8, q = 8 * (t / 32) + qi, m0 = 8 * grp;
            double a0 = v.x[m0 + u][q], a1 = v.x[m0 + u + 4][q];
            // X_mq = (delta - sum) / L_mm; a column beyond the row stays zero
            const int col = 8 * block(t / 32) + qi;
            a0 = (col == m0 + u ? 1.0 : 0.0) - a0;
            a1 = (col == m0 + u + 4 ? 1.0 : 0.0) - a1;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const double xm = __shfl_sync(0xffffffffu, (c < 4 ? a0 : a1) * v.inv[grp & 1][c], 8 * (c & 3) + qi);
                if (u == (c & 3)) (c < 4 ? a0 : a1) = xm;
                if (c < 4) a0 = u > c ? fma(-ld[c][m0 + u], xm, a0) : a0;
                a1 = u + 4 > c ? fma(-ld[c][m0 + u + 4], xm, a1) : a1;
            }
            v.x[m0 + u][q] = a0;
            v.x[m0 + u + 4][q] = a1;
        }
        named_sync(1, kDiagOwners);
        if (r / 8 > grp) {
            // (a branch per block: as a condition on each product the pipe took them all)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                if (j < nj && block(j) <= grp) {
                    double sum = w[j];
#pragma unroll
                    for (int c = 0; c < 8; ++c) sum = fma(ld[c][r], v.x[8 * grp + c][qi + 8 * j], sum);
                    w[j] = sum;
                }
        }
    }
    named_sync(1, kDiagOwners);
    // The rows of the scaled factor's inverse in digits, one exponent per row over all these CTAs: thread (row, 8
    // columns).  The panel's rows carry the scales.
    const int row = t % TS, part = t / TS;
    int f = -(1 << 28);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int q = 3 * part + c, col = 8 * block(q / 8) + q % 8;
        if (q < 8 * nj && col <= row) f = max(f, scaled_field(v.x[row][q], 0));
    }
    atomicMax(&v.smax[0][row], f);
    named_sync(1, kDiagOwners);
    if (t < TS) {
        f = v.smax[0][row];
        for (int rk = 1; rk < kDiagCtas; ++rk) st_cluster(mapa(&v.smax[rank][row], rk), f);
    }
    cluster_barrier();  // the last access to another CTA's shared memory
    const int e = scaled_row_exp(max(max(v.smax[1][row], v.smax[2][row]), v.smax[3][row]));
    if (rank == 1 && part == 0) g.dex[(size_t)b * TS + row] = e;
    if (part < nj) {
        unsigned long long d[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int q = 8 * part + c, col = 8 * block(part) + c;
            d[c] = to_digits(col <= row ? to_fixed(v.x[row][q], e) : 0);
        }
        unsigned char* o = g.dimg + (size_t)b * kDImg + block(part) * kDCore + row * 16;
        store_digits(d, [&](int i, uint4 x) { *reinterpret_cast<uint4*>(o + i * kDPlane) = x; });
    }
}

// four columns of all eight accumulators (NC columns apart), load and wait in one statement
template <int NC>
__device__ __forceinline__ void tmem_ld_acc4(uint32_t t, uint32_t (&r)[8][4])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%33];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%34];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12, %13, %14, %15}, [%35];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16, %17, %18, %19}, [%36];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20, %21, %22, %23}, [%37];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24, %25, %26, %27}, [%38];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%28, %29, %30, %31}, [%39];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[1][0]), "=r"(r[1][1]), "=r"(r[1][2]),
          "=r"(r[1][3]), "=r"(r[2][0]), "=r"(r[2][1]), "=r"(r[2][2]), "=r"(r[2][3]), "=r"(r[3][0]), "=r"(r[3][1]),
          "=r"(r[3][2]), "=r"(r[3][3]), "=r"(r[4][0]), "=r"(r[4][1]), "=r"(r[4][2]), "=r"(r[4][3]), "=r"(r[5][0]),
          "=r"(r[5][1]), "=r"(r[5][2]), "=r"(r[5][3]), "=r"(r[6][0]), "=r"(r[6][1]), "=r"(r[6][2]), "=r"(r[6][3]),
          "=r"(r[7][0]), "=r"(r[7][1]), "=r"(r[7][2]), "=r"(r[7][3])
        : "r"(t), "r"(t + NC), "r"(t + 2 * NC), "r"(t + 3 * NC), "r"(t + 4 * NC),
          "r"(t + 5 * NC), "r"(t + 6 * NC), "r"(t + 7 * NC)
        : "memory");
}

// The eight accumulators of one entry joined, in units of 2^(ea + eb - 55), rounded to the nearest.
// Accumulators 0 .. 4 are at most 2^22 (64 columns of at most 4 products of 2^14, the two with a top digit,
// which is at most 64, counting half), so adding 1.5 2^23 leaves the number in the low mantissa bits;
// pairs fit 32 bits.
__device__ __forceinline__ long long join_acc4(const uint32_t (&r)[8][4], int q)
{
    constexpr unsigned kMagic = 0x4b400000u;  // 1.5 2^23
    auto m = [&](int s) { return __float_as_uint(__uint_as_float(r[s][q]) + 12582912.0f); };
    auto f = [&](int s) { return (unsigned)__float2int_rn(__uint_as_float(r[s][q])); };
    const int v01 = (int)(m(0) * 256u + (m(1) - kMagic * 257u));
    const int v23 = (int)(m(2) * 256u + (m(3) - kMagic * 257u));
    const int v45 = (int)(m(4) * 256u + (f(5) - kMagic * 256u));
    const int v67 = (int)(f(6) * 256u + (f(7) + 4096u));
    long long x = (long long)v45 * 8 + (v67 >> 13);
    x = (long long)v23 * 524288 + x;
    return x + ((long long)v01 << 35);
}

// Panel of step k, one CTA per row pair: rows x (64 columns) times the inverted diagonal block, S_ik 2^-e by
// (2^-e L_kk)^-T with the diagonal's scales e, the
// products formed as above, the result rounded row by row to digits without passing through FP64
// (E's rows also to FP64, which the solve and the gradient read).  Thread (row m of the pair image,
// columns 16 cq .. 16 cq + 15).  The chain of loads, row maximum, digits, products, row maximum, digits
// bounds it; the loops over 8 columns stay rolled and read their input twice (the tile, the
// joined accumulators), since the unrolled form spent a third of its 30 us waiting for instructions.
constexpr int kPanelA = 0, kPanelB = kImg, kPanelTail = kImg + kDImg;
constexpr int kPanelThreads = 512;
constexpr int kPanelSmem = kPanelTail + 4 * 128 * 4 + 2 * TS * 4;

__global__ void __launch_bounds__(kPanelThreads, 1) digit_panel(int k, Dig g)
{
    extern __shared__ __align__(128) unsigned char sm[];
    int* smax = reinterpret_cast<int*>(sm + kPanelTail);  // [4][128]
    int* deb = smax + 512;                                // [64] exponents of the inverse's rows
    int* scale = deb + TS;                                // [64] diag_scale of the columns
    __shared__ uint64_t full, done;
    __shared__ uint32_t tptr;
    const int t = threadIdx.x, b = blockIdx.y, m = t & 127, cq = t >> 7, warp = t >> 5;
    const int q0 = (k + 1) / 2, nq = g.nt / 2 - q0;
    const bool isext = (int)blockIdx.x >= nq;
    const int pair = isext ? g.nt / 2 + (int)blockIdx.x - nq : q0 + (int)blockIdx.x;
    const int half = m >> 6, r = m & 63;
    const int blk = 2 * pair + half, eb = blk - g.nt;
    const bool valid = isext ? (g.ext != DIGIT_EXT_IDENTITY || eb <= k) : blk > k;
    launch_dependents();
    if (warp == 0) tmem_alloc(&tptr, 512);
    if (t == 0) {
        mbar_init(&full, 1);
        mbar_init(&done, 1);
        fence_mbar_init();
    }
    // The rows' column k is final before the diagonal block starts (its kernel waits for the update before it, and
    // this one starts after that wait), so their digits are made beside it (read from L2, where that update left
    // them); the inverted block comes after the wait.
    double* tile = nullptr;
    double v[16];
    if (t < TS)
        scale[t] = diag_scale(__ldcg(g.A + (size_t)b * g.strideA + (size_t)tile_index(k, k) * TILE_ELEMS + t * (TS + 1)));
    if (valid) {
        tile = (isext ? ext_tile(g, b, eb, k)
                      : g.A + (size_t)b * g.strideA + (size_t)tile_index(blk, k) * TILE_ELEMS) +
               r + TS * 16 * cq;
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = __ldcg(&tile[TS * c]);
    }
    __syncthreads();
    int f = -(1 << 28);
    if (valid)
#pragma unroll
        for (int c = 0; c < 16; ++c) f = max(f, scaled_field(v[c], scale[16 * cq + c]));
    smax[128 * cq + m] = f;
    __syncthreads();
    const int ea = scaled_row_exp(max(max(smax[m], smax[128 + m]), max(smax[256 + m], smax[384 + m])));
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        unsigned long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int col = 8 * h + c;
            w[c] = valid ? to_digits(to_fixed(__ldcg(&tile[TS * col]), ea + scale[16 * cq + col])) : 0;
        }
        unsigned char* o = sm + kPanelA + (2 * cq + h) * kCore + m * 16;
        store_digits(w, [&](int i, uint4 d) { *reinterpret_cast<uint4*>(o + i * kPlane) = d; });
    }
    fence_proxy_async();
    wait_prior();
    if (t == 0) {
        mbar_arrive_expect_tx(&full, kDImg);
        bulk_g2s(smem_u32(sm + kPanelB), g.dimg + (size_t)b * kDImg, kDImg, &full);
    }
    if (t < TS) deb[t] = g.dex[(size_t)b * TS + t];
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tptr;
    bool ok = true;
    if (t == 0) {
        bounded_wait(ok, &full, 0, g.err, g.waits);
        const uint64_t ad = smem_desc(smem_u32(sm + kPanelA), kCore, kGroupBytes);
        const uint64_t bd = smem_desc(smem_u32(sm + kPanelB), kDCore, kGroupBytes);
        if (ok)
            for (int kc = 0; kc < 4; ++kc)
                issue_products<TS>(tmem, ad + (uint64_t)kc * (2 * kCore >> 4), bd + (uint64_t)kc * (2 * kDCore >> 4),
                                   kPlane, kDPlane, kc == 0);
        mma_commit(&done);
    }
    __syncwarp();
    bounded_wait(ok, &done, 0, g.err, g.waits);
    if (!ok && t == 0) {  // the copy and the products, if they are under way
        mbar_wait(&full, 0, kWaits);
        mbar_wait(&done, 0, kWaits);
    }
    fence_after();
    __syncwarp();
    // this thread's entries in units of 2^(ea + deb[c] - 55), into the place of the rows' digits, and the row's largest
    long long* const mine = reinterpret_cast<long long*>(sm + kPanelA) + t;
    const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 16 * cq;
    int top = -(1 << 28);
#pragma unroll 1
    for (int h = 0; h < 4; ++h) {
        uint32_t acc[8][4];
        __syncwarp();
        tmem_ld_acc4<TS>(ta + 4 * h, acc);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const long long x = join_acc4(acc, c);
            mine[kPanelThreads * (4 * h + c)] = x;
            const int e = deb[16 * cq + 4 * h + c];
            if (x != 0 || e == kNonFinite) top = max(top, e + 64 - __clzll(x < 0 ? -x : x));
        }
    }
    smax[128 * cq + m] = top;  // its readers passed the barrier above the products
    __syncthreads();
    top = max(max(smax[m], smax[128 + m]), max(smax[256 + m], smax[384 + m]));
    const bool nonfinite = ea == kNonFinite || top > kNonFinite / 2;
    const int e = nonfinite ? kNonFinite : top < -(1 << 27) ? -1022 : top + ea - 55;
    const bool wide = isext && g.ext == DIGIT_EXT_ROWS;
    if (valid && cq == 0) g.ex[((size_t)b * dig_pairs(g) + pair) * 128 + m] = e;
    unsigned char* out = g.img + ((size_t)b * dig_pairs(g) + pair) * kImg + (size_t)m * 16;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        unsigned long long w[8];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            long long x[4];
            int sx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = 8 * h + 4 * q + c, de = deb[16 * cq + col];
                x[c] = mine[kPanelThreads * col];
                sx[c] = ea + de - 55;
                // X = x 2^(de - top + 54): |x| < 2^(top - de), so |X| < 2^54
                const int sh = de - top + 54;
                long long y = 0;
                if (!nonfinite) {
                    if (sh >= 0) y = x[c] << min(sh, 63);
                    else if (sh > -64) y = ((x[c] >> (-sh - 1)) + 1) >> 1;
                }
                w[4 * q + c] = to_digits(y);
            }
            if (wide) {
                double d[4];
                scaled_ints<4>(x, sx, 0, d);
#pragma unroll
                for (int c = 0; c < 4; ++c) tile[TS * (8 * h + 4 * q + c)] = d[c];
            }
        }
        unsigned char* o = out + (2 * cq + h) * kCore;
        if (valid) store_digits(w, [&](int i, uint4 d) { *reinterpret_cast<uint4*>(o + i * kPlane) = d; });
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// Update of step k: persistent CTAs over (pair, pair) jobs of 128 x 128 outputs, K = 64.  A job is four
// passes of 32 columns, whose eight accumulators take 256 tensor-memory columns: two passes are in flight (one
// 64-column pass after the other with 8 warps took 22 us a job).  Warp 17 works out the jobs and fetches, warp
// 16 issues the products, warps 0 .. 15 join a pass's accumulators and add them to the FP64 matrix while the
// next pass runs.
//
// A CTA takes its jobs in runs of up to kRun that share the first pair: its image stays in shared memory, and
// the second pair's comes in four pieces, each fetched as soon as the pass that used it is done, three passes
// ahead of the next (both images again for every job, and every warp working out the job: 11.1 us a job in a
// batch of 16 at nside 16, this 9.9).  Per job and SM the tensor cores need 8.7 k cycles, the FP64 pipe (one
// addition per output, 64 cycles per warp and partition) 8.2 k, the issue slots (about 80 instructions per
// output and thread, 20 to join, 25 to convert) 10 k; the matrix takes 256 KB of DRAM traffic, 5.0 of the 6.8 TB/s.
constexpr int kUpB = kImg, kUpSmem = 2 * kImg, kRun = 8;
constexpr int kUpWarps = 16, kUpThreads = (kUpWarps + 2) * 32, kPassCols = 32;

// job s of this CTA: whole rounds of kRun jobs per CTA, then the rest in equal runs; -1 past the last
__device__ __forceinline__ int up_at(int s, int njobs)
{
    const int G = gridDim.x, base = s / kRun * kRun * G, rest = njobs - base;
    if (rest <= 0) return -1;
    const int run = min(kRun, (rest + G - 1) / G), i = s % kRun, job = base + (int)blockIdx.x * run + i;
    return i < run && job < njobs ? job : -1;
}

// box of a piece: 32 rows of all digits and columns of one image
__device__ __forceinline__ void tensor_g2s(uint32_t dst, const CUtensorMap* map, int piece, int image, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(piece), "r"(8 * kDig * image), "r"(smem_u32(bar))
        : "memory");
}

struct UpJob {
    int b, kind, p, q;        // kind 0: A's trailing part, 1: E's rows, 2: V = M^T M; q: columns, p: rows
    int pa, pb;               // images
};

// The jobs of a launch: column pairs [q0, q0 + ncol) of the trailing part (ncol = 1 or all that are left), E's
// rows over the same columns, and with v the pairs of V
struct UpRange {
    int q0, ncol, npe, v;
    int a = 1;                // 0: E's rows alone
    int part = 0;             // of column pair q0, 1: the first half alone, 2: the second alone
};
__host__ __device__ inline int up_tri(const UpRange& u, int nq)
{
    const int m = nq - u.q0;
    return u.a == 0 ? 0 : u.ncol == 1 ? m : m * (m + 1) / 2;
}
__host__ __device__ inline int up_jobs(const UpRange& u, int nq)
{
    return (u.ncol > 0 ? up_tri(u, nq) + u.npe * u.ncol : 0) + (u.v ? u.npe * (u.npe + 1) / 2 : 0);
}

__device__ __forceinline__ UpJob up_job(const Dig& g, const UpRange& u, int per, int job)
{
    UpJob j;
    j.b = job / per;
    int l = job % per;
    const int nq = g.nt / 2, tri = u.ncol > 0 ? up_tri(u, nq) : 0;
    if (l < tri) {
        if (u.ncol == 1) {
            j.q = u.q0;
            j.p = u.q0 + l;
        } else {
            int I, J;
            tile_coords(l, I, J);
            j.q = u.q0 + J;
            j.p = u.q0 + I;
        }
        j.kind = 0;
        j.pa = j.p;
        j.pb = j.q;
        return j;
    }
    l -= tri;
    if (l < u.npe * u.ncol) {
        j.kind = 1;
        j.q = u.q0 + l % u.ncol;
        j.p = l / u.ncol;
        j.pa = nq + j.p;
        j.pb = j.q;
        return j;
    }
    l -= u.npe * u.ncol;
    tile_coords(l, j.p, j.q);
    j.kind = 2;
    j.pa = nq + j.p;
    j.pb = nq + j.q;
    return j;
}

// the passes of a job: halves [h0, h1) of the second pair, two parities each
__device__ __forceinline__ void up_halves(const UpRange& u, const UpJob& j, int k, int& h0, int& h1)
{
    h0 = (j.kind != 2 && 2 * j.q <= k) ? 1 : 0;      // the half with column k is not part of the update
    h1 = (j.kind == 2 && 2 * j.q + 1 > k) ? 1 : 2;
    if (j.kind != 2 && j.q == u.q0) {
        if (u.part == 1) h1 = 1;
        if (u.part == 2) h0 = 1;
    }
}

// a job's tile of the FP64 matrix, row block rb and column block cb (nullptr where the job does not touch it)
__device__ __forceinline__ double* up_tile(const Dig& g, const UpJob& j, int k, int rb, int cb)
{
    double* Ab = g.A + (size_t)j.b * g.strideA;
    if (j.kind == 0) return rb > k && rb >= cb ? Ab + (size_t)tile_index(rb, cb) * TILE_ELEMS : nullptr;
    if (j.kind == 1) return g.ext != DIGIT_EXT_IDENTITY || rb <= k ? ext_tile(g, j.b, rb, cb) : nullptr;
    return rb <= k && rb >= cb ? Ab + (size_t)tile_index(rb, cb) * TILE_ELEMS : nullptr;
}

// what a job's warps need, from the one thread that works it out (with a division or two and a root per job,
// 18 warps each for themselves took a tenth of the issue slots)
struct UpDesc {
    double* tile[2][2];       // by row block and column block; nullptr: not part of the job
    const int *ea, *eb;       // row exponents of the two pairs
    int i0, i1;               // passes; none: past the last job
    unsigned flip;            // sign of the products
    bool fresh;               // another first image than the job before
    bool start[2];            // by row block: V's row k starts here
};
constexpr int kUpDescs = 4;

__device__ __forceinline__ void up_desc(const Dig& g, const UpRange& u, const UpJob& j, int k, bool fresh, UpDesc& d)
{
    const int pairs = dig_pairs(g);
    int h0, h1;
    up_halves(u, j, k, h0, h1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int a = i & 1, b = i >> 1;
        d.tile[a][b] = b >= h0 && b < h1 ? up_tile(g, j, k, 2 * j.p + a, 2 * j.q + b) : nullptr;
    }
    d.ea = g.ex + ((size_t)j.b * pairs + j.pa) * 128;
    d.eb = g.ex + ((size_t)j.b * pairs + j.pb) * 128;
    d.i0 = 2 * h0;
    d.i1 = 2 * h1;
    d.flip = j.kind == 2 || g.ext == DIGIT_EXT_PRODUCT ? 0u : 0x80000000u;
    d.fresh = fresh;
    d.start[0] = j.kind == 2 && 2 * j.p == k;
    d.start[1] = j.kind == 2 && 2 * j.p + 1 == k;
}

// SETS: several sets of images per job (a product); a factorisation's step has one
template <bool SETS>
__global__ void __launch_bounds__(kUpThreads, 1)
    digit_update(int k, int njobs, int per, UpRange u, Dig g, const __grid_constant__ CUtensorMap map)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t afull[4], aempty[4], bfull[4], bempty[4], tfull[2], tempty[2], dfull[kUpDescs], dempty[kUpDescs], fin;
    __shared__ UpDesc desc[kUpDescs];
    __shared__ uint32_t tptr;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int nk = SETS ? g.nk : 1;
    launch_dependents();
    if (warp == 0) tmem_alloc(&tptr, 512);
    if (t == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(&afull[i], 1);
            mbar_init(&aempty[i], 1);
            mbar_init(&bfull[i], 1);
            mbar_init(&bempty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], kUpWarps);
        }
        for (int i = 0; i < kUpDescs; ++i) {
            mbar_init(&dfull[i], 1);
            mbar_init(&dempty[i], kUpWarps + 1);
        }
        mbar_init(&fin, 1);
        fence_mbar_init();
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tptr;
    bool ok = true;
    // (a constant: as a parameter the limit took 3 % of the update)
    auto wait = [&](uint64_t* bar, uint32_t parity) { bounded_wait(ok, bar, parity, g.err, kWaits); };
    // (the jobs are worked out before the wait for the kernel before this one, which precedes every access to memory)
    if (warp == kUpWarps + 1) {
        if (lane == 0) {
            uint32_t aphase = 0, bphase = 0;  // uses so far, mod 2: of A's and B's piece i in bit i
            // job s into its slot (i1 = 0 past the last)
            auto put = [&](int s, int job, const UpJob& j, bool fresh) {
                UpDesc& d = desc[s % kUpDescs];
                wait(&dempty[s % kUpDescs], ((s / kUpDescs) & 1) ^ 1);
                if (!ok) return;
                if (job >= 0) up_desc(g, u, j, k, fresh, d);
                else d.i0 = d.i1 = 0;
                mbar_arrive(&dfull[s % kUpDescs]);
            };
            int job = up_at(0, njobs), next = -1;
            UpJob j = up_job(g, u, per, max(job, 0)), n = j;
            const int pairs = dig_pairs(g);
            bool fresh = true, same = false;
            put(0, job, j, true);
            auto ahead = [&](int s) {  // the job after this one, s, into its slot
                next = up_at(s, njobs);
                n = up_job(g, u, per, max(next, 0));
                same = nk == 1 && next >= 0 && n.b == j.b && n.pa == j.pa;
                put(s, next, n, !same);
            };
            if (job >= 0) ahead(1);
            wait_prior();
            for (int s = 0; ok && job >= 0; ++s) {
                if (g.prefetch && next >= 0) {  // the next job's tiles on their way from DRAM
                    const UpDesc& d = desc[(s + 1) % kUpDescs];
#pragma unroll 1
                    for (int i = 0; i < 4; ++i)
                        if (d.tile[i & 1][i >> 1])
                            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(d.tile[i & 1][i >> 1]),
                                         "r"((uint32_t)(TILE_ELEMS * sizeof(double)))
                                         : "memory");
                }
                int h0, h1;
                up_halves(u, j, k, h0, h1);
                for (int ks = 0; ks < nk; ++ks) {
                    const int ia = ks * g.kim + j.b * pairs + j.pa, ib = g.im0 + ks * g.kim + j.b * pairs + j.pb;
                    auto piece = [&](int i) {
                        wait(&bempty[i], ((bphase >> i) & 1) ^ 1);
                        if (!ok) return;
                        bphase ^= 1u << i;
                        mbar_arrive_expect_tx(&bfull[i], kPiece);
                        tensor_g2s(smem_u32(sm + kUpB + i * kPiece), &map, i, ib, &bfull[i]);
                    };
                    auto rows = [&]() {
                        const unsigned char* a = g.img + (size_t)ia * kImg;
                        for (int kc = 0; kc < 4; ++kc) {
                            wait(&aempty[kc], ((aphase >> kc) & 1) ^ 1);
                            if (!ok) return;
                            aphase ^= 1u << kc;
                            mbar_arrive_expect_tx(&afull[kc], 2 * kCore);
                            bulk_g2s(smem_u32(sm + 2 * kc * kCore), a + 2 * kc * kCore, 2 * kCore, &afull[kc]);
                        }
                    };
                    // in the order in which the places become free
                    const bool first = s == 0 && ks == 0;
                    piece(2 * h0);
                    if (first) rows();
                    for (int i = 2 * h0 + 1; i < 2 * h1 - 1; ++i) piece(i);
                    if (!first && fresh) rows();
                    piece(2 * h1 - 1);
                }
                job = next;
                j = n;
                fresh = !same;
                if (job >= 0) ahead(s + 2);
            }
            if (!ok)  // the copies under way
                for (int i = 0; i < 4; ++i) {
                    mbar_wait(&afull[i], ((aphase >> i) & 1) ^ 1, kWaits);
                    mbar_wait(&bfull[i], ((bphase >> i) & 1) ^ 1, kWaits);
                }
        }
        __syncwarp();
    } else if (warp == kUpWarps) {
        if (lane == 0) {
            uint32_t aphase = 0, bphase = 0, pass = 0;
            for (int s = 0;; ++s) {
                const UpDesc& d = desc[s % kUpDescs];
                wait(&dfull[s % kUpDescs], (s / kUpDescs) & 1);
                const int i0 = d.i0, i1 = ok ? d.i1 : 0;
                if (i1 == 0) break;
                const bool fresh = d.fresh;
                const UpDesc& n = desc[(s + 1) % kUpDescs];  // put there before this job's images were fetched
                wait(&dfull[(s + 1) % kUpDescs], ((s + 1) / kUpDescs) & 1);
                const bool last = n.i1 == 0 || n.fresh;
                for (int ks = 0; ks < nk; ++ks) {
                    for (int i = i0; i < i1; ++i, ++pass) {
                        const uint32_t buf = pass & 1;
                        wait(&tempty[buf], ((pass >> 1) & 1) ^ 1);
                        wait(&bfull[i], (bphase >> i) & 1);
                        bphase ^= 1u << i;
                        fence_after();
                        const uint64_t ad = smem_desc(smem_u32(sm), kCore, kGroupBytes);
                        const uint64_t bd = smem_desc(smem_u32(sm + kUpB + i * kPiece), kPieceCore, kGroupBytes);
                        for (int kc = 0; kc < 4; ++kc) {
                            if (fresh && i == i0) wait(&afull[kc], aphase);
                            issue_products<kPassCols>(tmem + 256 * buf, ad + (uint64_t)kc * (2 * kCore >> 4),
                                                      bd + (uint64_t)kc * (2 * kPieceCore >> 4), kPlane, kPieceRow,
                                                      kc == 0);
                            if (last && i == i1 - 1) mma_commit(&aempty[kc]);
                        }
                        mma_commit(&bempty[i]);
                        mma_commit(&tfull[buf]);
                    }
                    if (fresh) aphase ^= 1;
                }
                mbar_arrive(&dempty[s % kUpDescs]);
            }
            if (!ok) {  // the products under way
                mma_commit(&fin);
                mbar_wait(&fin, 0, kWaits);
            }
        }
        __syncwarp();
    } else {
        wait_prior();
        const int m = 32 * (warp & 3) + lane, c4 = warp >> 2;  // row of the pair image, 8-column group of the pass
        const int half = m >> 6, r = m & 63;
        int s = 0, i = 0, i0 = 0, i1 = 0, ks = 0;
        const int *ea = nullptr, *eb = nullptr;  // of this thread's row, of the job's columns
        // A pass's entries of the matrix (the thread's eight columns from dst on; nullptr: not part of it) are
        // loaded four at a time as soon as the pass before is done with the registers.
        double* dst = nullptr;
        double old[8];
        auto open_job = [&]() {  // false: no more jobs
            wait(&dfull[s % kUpDescs], (s / kUpDescs) & 1);
            const UpDesc& d = desc[s % kUpDescs];
            i0 = d.i0;
            i1 = ok ? d.i1 : 0;
            ea = d.ea + m;
            eb = d.eb + 8 * c4;
            i = i0;
            ks = 0;
            return i1 != 0;
        };
        auto open_pass = [&]() {
            dst = desc[s % kUpDescs].tile[half][i >> 1];
            if (dst != nullptr) dst += r + TS * (32 * (i & 1) + 8 * c4);
        };
        bool more = __all_sync(0xffffffffu, open_job());  // a warp leaves as a whole
        if (more) {
            open_pass();
            const bool read = dst != nullptr && !desc[s % kUpDescs].start[half];
#pragma unroll
            for (int c = 0; c < 8; ++c) old[c] = read ? dst[TS * c] : 0.0;
        }
        for (uint32_t pass = 0; more; ++pass) {
            const uint32_t buf = pass & 1;
            const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 256 * buf + 8 * c4;
            double* const out = dst;
            const unsigned flip = desc[s % kUpDescs].flip;
            const int e = ea[ks * g.kex] - 55;
            const int4* const ec = reinterpret_cast<const int4*>(eb + ks * g.kex + 32 * i);
            const int4 e0 = ec[0], e1 = ec[1];
            const int se[8] = {e + e0.x, e + e0.y, e + e0.z, e + e0.w, e + e1.x, e + e1.y, e + e1.z, e + e1.w};
            if (++i == i1) {
                if (SETS && ++ks < nk) {
                    i = i0;
                } else {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&dempty[s % kUpDescs]);
                    ++s;
                    more = open_job();
                }
            }
            bool read = false;
            if (more) {
                open_pass();
                read = dst != nullptr && !desc[s % kUpDescs].start[half];
            }
            wait(&tfull[buf], (pass >> 1) & 1);
            fence_after();
            more = __all_sync(0xffffffffu, more);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                uint32_t acc[8][4];
                tmem_ld_acc4<kPassCols>(ta + 4 * q, acc);
                if (q == 1) {
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tempty[buf]);
                }
                if (out != nullptr) {
                    long long x[4];
                    int sx[4];
                    double d[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        x[c] = join_acc4(acc, c);
                        sx[c] = se[4 * q + c];
                    }
                    scaled_ints<4>(x, sx, flip, d);
#pragma unroll
                    for (int c = 0; c < 4; ++c) out[TS * (4 * q + c)] = old[4 * q + c] + d[c];
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) old[4 * q + c] = read ? dst[TS * (4 * q + c)] : 0.0;
                __syncwarp();
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// Images of a dense operand's row pairs for K blocks k0, k0 + 1, ..: grid (row pairs, K blocks).  Element
// (row, k): kind 0 at k ld + row (B of a product, row-major), kind 1 at row ld + k (A), kind 2 in 64 x 64 tiles (k / 64, row / 64) of nt to a
// row, element (r, c) at r + 64 c.  Column k is scaled by 2^(-sign scale[k]).  Thread (row, 16 columns), as in the panel.
__global__ void __launch_bounds__(kPanelThreads) digit_slice(int kind, int ld, int k0, int first, const double* __restrict__ src,
                                                             const int* __restrict__ scale, int sign, Dig g)
{
    __shared__ int smax[4][128];
    const int t = threadIdx.x, m = t & 127, cq = t >> 7, pair = blockIdx.x, nt = ld / TS;
    const int row = 128 * pair + m;
    const int kb = k0 + blockIdx.y;
    auto at = [&](int c) {
        const int k = TS * kb + c;
        return kind == 0   ? src[(size_t)k * ld + row]
               : kind == 1 ? src[(size_t)row * ld + k]
                           : src[((size_t)kb * nt + row / TS) * TILE_ELEMS + c + TS * (m % TS)];
    };
    auto shift = [&](int c) { return sign * scale[TS * kb + c]; };
    int f = -(1 << 28);
#pragma unroll
    for (int c = 0; c < 16; ++c) f = max(f, scaled_field(at(16 * cq + c), shift(16 * cq + c)));
    smax[cq][m] = f;
    __syncthreads();
    const int e = scaled_row_exp(max(max(smax[0][m], smax[1][m]), max(smax[2][m], smax[3][m])));
    const size_t p = first + pair;
    if (cq == 0) g.ex[blockIdx.y * g.kex + p * 128 + m] = e;
    unsigned char* out = g.img + blockIdx.y * g.kimg + p * kImg + (size_t)m * 16;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        unsigned long long w[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int col = 16 * cq + 8 * h + c;
            w[c] = to_digits(to_fixed(at(col), e + shift(col)));
        }
        unsigned char* o = out + (2 * cq + h) * kCore;
        store_digits(w, [&](int i, uint4 d) { *reinterpret_cast<uint4*>(o + i * kPlane) = d; });
    }
}

// Scales of the columns of a symmetric matrix C (ld x ld): C_ik 2^-(half[i] + scale[k]) is at most 1.  half[i] is the
// diagonal's (of a row without one, its largest entry's), and scale[k] = max_i of what the entries need, half[k] but
// for a rounding where C is positive semidefinite.  A column of zeros gets kNoScale, which puts what it meets below
// every other entry.  One CTA per row.
constexpr int kNoScale = -(1 << 14);

__device__ __forceinline__ int cta_max(int v)
{
    __shared__ int red[kPanelThreads / 32];
    v = __reduce_max_sync(0xffffffffu, v);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = v;
    __syncthreads();
    return __reduce_max_sync(0xffffffffu, red[threadIdx.x % (kPanelThreads / 32)]);
}

__global__ void __launch_bounds__(kPanelThreads) half_scales(int ld, const double* __restrict__ C, int* __restrict__ half)
{
    const double* row = C + (size_t)blockIdx.x * ld;
    double d = row[blockIdx.x];
    if (exp_field(d) == 0) {  // (the same for every thread)
        int f = 0;
        for (int i = threadIdx.x; i < ld; i += kPanelThreads) f = max(f, exp_field(row[i]));
        d = __hiloint2double(cta_max(f) << 20, 0);
    }
    if (threadIdx.x == 0) half[blockIdx.x] = diag_scale(d);
}

__global__ void __launch_bounds__(kPanelThreads) column_scales(int ld, const double* __restrict__ C, const int* __restrict__ half,
                                                              int* __restrict__ scale)
{
    const double* row = C + (size_t)blockIdx.x * ld;
    int f = kNoScale;
    for (int i = threadIdx.x; i < ld; i += kPanelThreads) {
        const int x = exp_field(row[i]);
        if (x) f = max(f, x - 1022 - half[i]);
    }
    f = cta_max(f);
    if (threadIdx.x == 0) scale[blockIdx.x] = f;
}

}  // namespace

// the images at base for tensor copies of their pieces: (512 bytes, 4 pieces, 56 digits of 8 columns per image)
static int image_map(cg_ctx* ctx, CUtensorMap* map, void* base, size_t images)
{
    static const auto encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(f);
    }();
    const cuuint64_t dims[3] = {kPieceRow / 8, 4, (cuuint64_t)images * 8 * kDig}, strides[2] = {kPieceRow, kPlane};
    const cuuint32_t box[3] = {kPieceRow / 8, 1, 8 * kDig}, step[3] = {1, 1, 1};
    if (!encode || encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, base, dims, strides, box, step,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        ctx->err = "cuTensorMapEncodeTiled: no tensor map for the digit images";
        return CG_ERR_CUDA;
    }
    return CG_OK;
}

size_t digit_bytes(int nt, int ne)
{
    const size_t pairs = (size_t)(nt + ne) / 2;
    return 2 * pairs * (kImg + 128 * sizeof(int)) + kDImg + TS * sizeof(int);
}

static int launch_update(cg_ctx* ctx, int B, int k, const UpRange& u, const Dig& g, const CUtensorMap& map, int ctas,
                         cudaStream_t s)
{
    const int per = up_jobs(u, g.nt / 2);
    if (per <= 0) return CG_OK;
    return launch(ctx, digit_update<false>, dim3((unsigned)std::min<long long>((long long)per * B, ctas)), kUpThreads, kUpSmem, 1, s,
                  k, per * B, per, u, g, map);
}

// The factorisation's chain (diagonal block, panel, the update of the next column pair) beside the rest of
// the update of the step before, on a second stream and on all but `reserve` SMs: the reserve that makes the
// longer of the two shortest, or 0 where one after the other is as fast.  Per SM a job takes about 10 us and a
// panel's CTA 12, the update of one pair 8, a diagonal step 30; a saving below 3 % is left.  One factorisation at
// nside 16 with its harmonics: 3.94 ms one after the other, 3.16 beside when this came in, 2.16 now; sixteen of them
// 14.94 -> 14.43 ms with the line at 3 % instead of 7 (14.10 at 2 %, but eight without harmonics 3.57 -> 3.63).
static int chain_reserve(const cg_ctx* ctx, int B, int nq, int npe, int v)
{
    const UpRange all = {0, nq, npe, v}, one = {0, 1, npe, 0};
    const double sms = ctx->sm_count, col = (double)up_jobs(one, nq) * B, jobs = (double)up_jobs(all, nq) * B;
    auto waves = [](double n, double s) { return std::max(1.0, std::ceil(n / s)); };
    const double serial = 30 + 12 * waves(col, sms) + 10 * waves(jobs, sms) + 6;
    double best = 0.97 * serial;
    int reserve = 0;
    for (int r = 8; r <= ctx->sm_count / 2; r += 8) {
        const double chain = 30 * waves((double)kDiagCtas * B, r) + 20 * waves(col, r) + 8;
        const double t = std::max(chain, 10 * waves(jobs - col, sms - r) + 4);
        if (t < best) {
            best = t;
            reserve = r;
        }
    }
    return reserve;
}

static bool chain_streams(cg_ctx* ctx)
{
    if (!ctx->aux && cudaStreamCreateWithFlags(&ctx->aux, cudaStreamNonBlocking) != cudaSuccess) ctx->aux = nullptr;
    bool ok = ctx->aux != nullptr;
    for (cudaEvent_t& e : ctx->ev_chain)
        if (ok && !e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            ok = false;
        }
    if (!ok) cudaGetLastError();
    return ok;
}

void digit_free(cg_ctx* ctx)
{
    if (ctx->aux) {
        cudaStreamSynchronize(ctx->aux);
        cudaStreamDestroy(ctx->aux);
        ctx->aux = nullptr;
    }
    for (cudaEvent_t& e : ctx->ev_chain) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
}

int digit_factor(cg_ctx* ctx, int B, int nt, int ne, int ext, double* A, size_t strideA, double* E,
                 size_t strideE, double* diag, int* status, unsigned char* work, int* err, cudaStream_t s)
{
    const size_t pairs = (size_t)(nt + ne) / 2;
    const int nq = nt / 2, v = ext == DIGIT_EXT_IDENTITY ? 1 : 0;
    Dig g;
    g.nt = nt;
    g.ne = ne;
    g.ext = ext;
    g.A = A;
    g.E = E;
    g.strideA = strideA;
    g.strideE = strideE;
    g.nk = 1;
    g.kimg = g.kex = 0;
    g.kim = 0;
    // 2 to 5 % of a factorisation that exceeds L2 (129 MB); 1 % lost on one that does not
    g.prefetch = sizeof(double) * B * (strideA + strideE) > ((size_t)100 << 20);
    // two sets of images, for the steps in turn where the update of one runs beside the panel of the next
    unsigned char* const img[2] = {work, work + (size_t)B * pairs * kImg};
    CUtensorMap map;
    if (int rc = image_map(ctx, &map, work, 2 * B * pairs)) return rc;
    g.dimg = img[1] + (size_t)B * pairs * kImg;
    int* const ex[2] = {reinterpret_cast<int*>(g.dimg + (size_t)B * kDImg),
                        reinterpret_cast<int*>(g.dimg + (size_t)B * kDImg) + (size_t)B * pairs * 128};
    g.dex = ex[1] + (size_t)B * pairs * 128;
    g.err = err;
    g.waits = ctx->no_waits ? 0 : kWaits;
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DiagShared)));
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmem));
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_update<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpSmem));
    bool rest = false;  // an update on the second stream that the caller's stream has not waited for
    for (int k = 0; k < nt; ++k) {
        const int q0 = (k + 1) / 2, m = nq - q0, npe = v ? k / 2 + 1 : ne / 2;
        g.img = img[0];
        g.ex = ex[0];
        g.im0 = 0;
        if (int rc = launch(ctx, digit_diag, dim3(kDiagCtas * B), kDiagThreads, sizeof(DiagShared), kDiagCtas, s, k, g, diag, status))
            return rc;
        if (m + npe == 0) continue;
        const int reserve = m > 1 ? chain_reserve(ctx, B, m, npe, v) : 0;
        const bool beside = reserve > 0 && chain_streams(ctx);
        if (rest && !beside) {
            CG_CUDA_TRY(ctx, cudaStreamWaitEvent(s, ctx->ev_chain[1], 0));
            rest = false;
        }
        if (beside || rest) {
            g.img = img[k & 1];
            g.ex = ex[k & 1];
            g.im0 = (k & 1) * B * (int)pairs;
        }
        if (int rc = launch(ctx, digit_panel, dim3(m + npe, B), kPanelThreads, kPanelSmem, 1, s, k, g)) return rc;
        if (!beside) {
            if (int rc = launch_update(ctx, B, k, {q0, m, npe, v}, g, map, ctx->sm_count, s)) return rc;
            continue;
        }
        CG_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_chain[0], s));
        CG_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->aux, ctx->ev_chain[0], 0));
        // the next column pair needs the rest of the step before
        if (rest) CG_CUDA_TRY(ctx, cudaStreamWaitEvent(s, ctx->ev_chain[1], 0));
        // Step k + 1 needs column k + 1 alone.  Where that is the first half of the pair, the second goes with the rest:
        // the update in the chain is two passes in every step (one factorisation at nside 16: 2545 -> 2495 us)
        const bool split = k % 2 == 1;
        if (int rc = launch_update(ctx, B, k, {q0, 1, npe, 0, 1, split ? 1 : 0}, g, map, ctx->sm_count, s)) return rc;
        const UpRange left = split ? UpRange{q0, m, npe, v, 1, 2} : UpRange{q0 + 1, m - 1, npe, v};
        if (int rc = launch_update(ctx, B, k, left, g, map, ctx->sm_count - reserve, ctx->aux)) return rc;
        CG_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_chain[1], ctx->aux));
        rest = true;
    }
    if (rest) CG_CUDA_TRY(ctx, cudaStreamWaitEvent(s, ctx->ev_chain[1], 0));
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int digit_selftest_timeout(cg_ctx* ctx, int* host_status)
{
    const int nt = 4;
    const size_t tiled = tiled_elems(nt);
    double *A = nullptr, *diag = nullptr;
    unsigned char* work = nullptr;
    int* st = nullptr;
    cudaStream_t s = ctx->stream;
    int rc = CG_OK, h[2] = {0, 0};
    if (cudaMalloc((void**)&A, 2 * tiled * sizeof(double)) != cudaSuccess ||
        cudaMalloc((void**)&diag, nt * TS * sizeof(double)) != cudaSuccess ||
        cudaMalloc((void**)&work, digit_bytes(nt, nt)) != cudaSuccess || cudaMalloc((void**)&st, sizeof h) != cudaSuccess) {
        cudaGetLastError();
        ctx->err = "device allocation failed";
        rc = CG_ERR_ALLOC;
    }
    if (!rc && cudaMemsetAsync(st, 0, sizeof h, s) != cudaSuccess) rc = CG_ERR_CUDA;
    if (!rc) rc = fp64_identity_rows(ctx, 2, nt, A, tiled, s);  // the matrix and E's rows
    if (!rc) {
        ctx->no_waits = true;
        rc = digit_factor(ctx, 1, nt, nt, DIGIT_EXT_IDENTITY, A, tiled, A + tiled, tiled, diag, st, work, st + 1, s);
        ctx->no_waits = false;
    }
    if (!rc) {
        cudaError_t e = cudaMemcpyAsync(h, st, sizeof h, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { ctx->err = cudaGetErrorString(e); rc = CG_ERR_CUDA; }
    }
    cudaFree(A);
    cudaFree(diag);
    cudaFree(work);
    cudaFree(st);
    *host_status = h[1] ? CG_ERR_TIMEOUT : CG_OK;
    return rc;
}

// K blocks whose images are held at once
static int gemm_chunk(int nt) { return std::min(nt, 16); }

size_t digit_gemm_bytes(int nt) { return (size_t)gemm_chunk(nt) * nt * (kImg + 128 * sizeof(int)); }

int digit_scales(cg_ctx* ctx, int ld, const double* C, int* scale, cudaStream_t s)
{
    half_scales<<<ld, kPanelThreads, 0, s>>>(ld, C, scale + ld);
    column_scales<<<ld, kPanelThreads, 0, s>>>(ld, C, scale + ld, scale);
    count_launch(ctx, 2);
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

int digit_gemm(cg_ctx* ctx, int nt, const double* A, const double* Bm, bool tilesB, double* out, const int* scale, int sign,
               unsigned char* work, int* err, cudaStream_t s)
{
    const int nq = nt / 2, chunk = gemm_chunk(nt), ld = nt * TS;
    Dig g = {};
    g.nt = g.ne = nt;
    g.ext = DIGIT_EXT_PRODUCT;
    g.A = g.E = out;
    g.kimg = (size_t)nt * kImg;
    g.kex = (size_t)nt * 128;
    g.kim = nt;
    g.img = work;
    g.ex = reinterpret_cast<int*>(work + chunk * g.kimg);
    g.err = err;
    g.waits = ctx->no_waits ? 0 : kWaits;
    CG_CUDA_TRY(ctx, cudaFuncSetAttribute(digit_update<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUpSmem));
    CUtensorMap map;
    if (int rc = image_map(ctx, &map, work, (size_t)chunk * nt)) return rc;
    const UpRange u = {0, nq, nq, 0, 0};
    const int per = up_jobs(u, nq);
    for (int k0 = 0; k0 < nt; k0 += chunk) {
        g.nk = std::min(chunk, nt - k0);
        digit_slice<<<dim3(nq, g.nk), kPanelThreads, 0, s>>>(tilesB ? 2 : 0, ld, k0, 0, Bm, scale, -sign, g);
        digit_slice<<<dim3(nq, g.nk), kPanelThreads, 0, s>>>(1, ld, k0, nq, A, scale, sign, g);
        digit_update<true><<<std::min(per, ctx->sm_count), kUpThreads, kUpSmem, s>>>(-1, per, per, u, g, map);
        count_launch(ctx, 3);
    }
    CG_CUDA_TRY(ctx, cudaGetLastError());
    return CG_OK;
}

}  // namespace cg
