// The packed pair arithmetic of the exact passes against CUDA's correctly rounded functions.
// Prints the number of mismatches of each check.
#include <cstdio>

#include "sphx_internal.cuh"

using namespace sphx;

__device__ __forceinline__ uint64_t mix(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// a float of random sign and significand with exponent in [-span, span]
__device__ __forceinline__ float rnd(uint64_t i, int span) {
    const uint64_t h = mix(i);
    const uint32_t e = (uint32_t)(127 + (int)((h >> 24) % (2 * span + 1)) - span);
    return __uint_as_float((uint32_t)(h >> 60 & 1) << 31 | e << 23 | (uint32_t)(h & 0x7fffff));
}

// every float x in [0, 2^86]: sqrt2_exact(x) == sqrt(x), and rcp2_exact of the root == its
// reciprocal wherever the root lies in [2^-40, 2^40]
__global__ void k_roots(PairLits k, unsigned long long* bad) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 2;
    const float a = __uint_as_float(i), b = __uint_as_float(i + 1);
    if (!(b <= 0x1p86f)) return;
    F2 h, ns;
    const F2 s = sqrt2_exact(k, f2(a, b), h, ns);
    const float2 u = upk2(s.v), n = upk2(ns.v);
    const float r[2] = {__fsqrt_rn(a), __fsqrt_rn(b)};
    if (u.x != r[0] || u.y != r[1] || n.x != -r[0] || n.y != -r[1]) atomicAdd(bad, 1ull);
    const float2 y = upk2(rcp2_exact(k, ns, h * F2{k.p2p21}).v);
    const float q[2] = {y.x, y.y};
    for (int c = 0; c < 2; ++c)
        if (r[c] >= 0x1p-40f && r[c] <= 0x1p40f && q[c] != __frcp_rn(r[c])) atomicAdd(bad + 1, 1ull);
}

// quotients by a shared reciprocal: random ones, divisors of all-ones significand, and every
// significand of the dividend for the largest significand of the divisor
__global__ void k_quotients(unsigned long long* bad) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    float a = rnd(2 * i, 60), b = fabsf(rnd(2 * i + 1, 20));
    if ((i & 3) == 0) b = __uint_as_float(__float_as_uint(b) | 0x7fffff);
    if ((i & 3) == 1) a = __uint_as_float(0x3f000000u + (uint32_t)(i >> 2)), b = 0x1.fffffep-1f;
    const float y = __frcp_rn(b);
    const float2 q = upk2(div_rcp2(f2(a, -a), f2(-b), f2(y)).v);
    if (q.x != __fdiv_rn(a, b) || q.y != __fdiv_rn(-a, b)) atomicAdd(bad, 1ull);
}

// sums of products in a loop: pmul keeps the product's own rounding
__global__ void k_products(PairLits k, unsigned long long* bad) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    __shared__ float w[256];
    w[threadIdx.x] = rnd(i + 9, 3);
    __syncthreads();
    const float a = rnd(4 * i, 3), b = rnd(4 * i + 1, 3), c = rnd(4 * i + 2, 3);
    const F2 A = f2(a, b), C = f2(c), neg0{k.neg0};
    F2 acc = f2(0.0f);
    float s = 0.0f, t = 0.0f;
    for (int j = 0; j < 8; ++j) {
        const float v = w[(threadIdx.x * 7 + j * 5) & 255];
        acc = acc + pmul(f2(v) * A, C, neg0);
        s = __fadd_rn(s, __fmul_rn(__fmul_rn(v, a), c));
        t = __fadd_rn(t, __fmul_rn(__fmul_rn(v, b), c));
    }
    const float2 u = upk2(acc.v);
    if (u.x != s || u.y != t) atomicAdd(bad, 1ull);
}

int main() {
    sphx_params p{};
    p.smoothing_length = 0.02f;
    p.neighbor_search_radius = 0.04f;
    StepConst c{};
    step_const_from_params(p, 1, SPHX_KERNEL_CUBIC_SPLINE, SPHX_MODE_EXACT, 125, c);
    unsigned long long* bad;
    cudaMallocManaged(&bad, 4 * sizeof(*bad));
    for (int k = 0; k < 4; ++k) bad[k] = 0;
    k_roots<<<1u << 22, 256>>>(c.lit, bad);  // every bit pattern, two a thread
    k_quotients<<<1u << 18, 256>>>(bad + 2);
    k_products<<<1u << 14, 256>>>(c.lit, bad + 3);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    printf("roots %llu reciprocals %llu quotients %llu products %llu\n", bad[0], bad[1], bad[2], bad[3]);
    return 0;
}
