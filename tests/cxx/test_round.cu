// root and quotient (cg_round.cuh) against sqrtf and divisions: prints the number of differences of each sweep.
#include <cstdio>
#include <cstdint>

#include "../../cosmopp_gb300/csrc/cg_round.cuh"

// every float of [2^-60, 2^60]: the root and its reciprocal, and `rare` for a root with a significand of ones alone
__global__ void sweep_roots(unsigned first, unsigned last, unsigned long long* bad)
{
    unsigned long long n = 0;
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = first + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i <= last; i += step) {
        const float v = __uint_as_float((unsigned)i), want = __fsqrt_rn(v);
        float d, rd;
        bool rare = false;
        cg::root(v, d, rd, rare);
        const bool ones = (__float_as_uint(want) & 0x7fffffu) == 0x7fffffu;
        if (__float_as_uint(d) != __float_as_uint(want) || rare != ones) ++n;
        if (!rare && __float_as_uint(rd) != __float_as_uint(__fdiv_rn(1.f, want))) ++n;
    }
    if (n) atomicAdd(bad, n);
}

// what is not in that range is left to the library
__global__ void edges(unsigned long long* bad)
{
    const float out[] = {0.f, -0.f, -1.f, 0x1.fffffep-61f, 0x1.000002p60f, 1e-45f, 3e38f, -3e38f,
                         __uint_as_float(0x7f800000u), __uint_as_float(0xff800000u), __uint_as_float(0x7fc00000u)};
    for (float v : out) {
        float d, rd;
        bool rare = false;
        cg::root(v, d, rd, rare);
        if (!rare) atomicAdd(bad, 1ull);
        rare = false;
        cg::quotient(v, 1.f, 1.f, rare);
        if (v != 0.f && v != -1.f && !rare) atomicAdd(bad, 1ull);
        rare = false;
        cg::quotient(1.f, v, 1.f, rare);
        if (!rare) atomicAdd(bad, 1ull);
    }
}

__device__ unsigned mix(unsigned long long x)
{
    x = (x ^ (x >> 31)) * 0x7fb5d329728ea185ull;
    x = (x ^ (x >> 27)) * 0x81dadef4bc2dd44dull;
    return (unsigned)(x >> 32);
}

// every significand of d but that of ones, by `per` numerators each: random ones, and those next to d, to a power of
// two and to the end of their binade
__global__ void sweep_quotients(unsigned per, unsigned long long* bad)
{
    unsigned long long n = 0;
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= 0x7fffffu) return;
    for (unsigned k = 0; k < per; ++k) {
        const unsigned h = mix(((unsigned long long)m << 32) | (2 * k)), x = mix(((unsigned long long)m << 32) | (2 * k + 1));
        const unsigned ed = 127 - 30 + h % 60, ev = 127 - 60 + (h >> 8) % 120;
        unsigned mv = x & 0x7fffffu;
        if (k % 8 == 5) mv = (m + (x & 15) - 8) & 0x7fffffu;
        if (k % 8 == 6) mv = x & 15;
        if (k % 8 == 7) mv = 0x7fffffu - (x & 15);
        const float d = __uint_as_float((ed << 23) | m), v = __uint_as_float((x & 0x80000000u) | (ev << 23) | mv);
        bool rare = false;
        const float q = cg::quotient(v, d, __frcp_rn(d), rare);
        if (rare || __float_as_uint(q) != __float_as_uint(__fdiv_rn(v, d))) ++n;
        const float z = cg::quotient(0.f, d, __frcp_rn(d), rare);
        if (rare || z != 0.f) ++n;
    }
    if (n) atomicAdd(bad, n);
}

int main()
{
    unsigned long long* d = nullptr;
    unsigned long long h[3] = {1, 1, 1};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
    sweep_roots<<<1024, 256>>>((127u - 60) << 23, (127u + 60) << 23, d);
    edges<<<1, 1>>>(d + 1);
    sweep_quotients<<<(1u << 23) / 256, 256>>>(256, d + 2);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
