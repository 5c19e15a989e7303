// Counts where the helpers of csrc/rounding.cuh differ from the IEEE operations: rcp_rn and
// sqrt_mid for every mantissa at several exponents, div_by for random operands (a quarter of the
// divisors with mantissas near all ones).  Prints four counts: reciprocal, root, quotient, CUDA error.
#include <cstdint>
#include <cstdio>

#include "rounding.cuh"

__global__ void mantissas(unsigned long long* bad, int e)
{
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;            // two binades: 2^24 values
    const float x = __uint_as_float(((uint32_t)(127 + e) << 23) + m);
    if (sysmat::rcp_rn(x) != __frcp_rn(x) || sysmat::rcp_rn(-x) != __frcp_rn(-x)) atomicAdd(&bad[0], 1ull);
    if (sysmat::sqrt_mid(x) != __fsqrt_rn(x)) atomicAdd(&bad[1], 1ull);
}

__global__ void quotients(unsigned long long* bad, uint64_t seed)
{
    uint64_t s = seed + (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull;
    unsigned long long n = 0;
    for (int i = 0; i < 1024; ++i) {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;                         // xorshift (Marsaglia 2003)
        const uint32_t u = (uint32_t)s, v = (uint32_t)(s >> 32);
        const float a = __uint_as_float((u & 0x807fffffu) | ((107 + (u >> 23) % 40) << 23));
        const uint32_t mb = (i & 3) ? (v & 0x007fffffu) : (0x007fffffu - (v & 31u));
        const float b = __uint_as_float((v & 0x80000000u) | mb | ((107 + (v >> 23 & 255u) % 40) << 23));
        n += sysmat::div_by(a, b, sysmat::rcp_rn(b)) != __fdiv_rn(a, b);
    }
    if (n) atomicAdd(&bad[2], n);
}

int main()
{
    unsigned long long *bad, h[3] = {1, 1, 1};
    cudaMalloc(&bad, sizeof(h));
    cudaMemset(bad, 0, sizeof(h));
    for (int e : {-60, -18, -17, -1, 0, 1, 12, 40}) mantissas<<<1 << 16, 256>>>(bad, e);
    for (uint64_t r = 1; r <= 4; ++r) quotients<<<4096, 256>>>(bad, r * 0x1234567ull);
    cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost);
    std::printf("%llu %llu %llu %d\n", h[0], h[1], h[2], (int)cudaGetLastError());
    return 0;
}
