// Largest distance in units of the last place between rcp64 and sqrt64 of csrc/rounding.cuh and the IEEE
// operations, over random doubles whose float value is normal (2^-125 .. 2^125), both signs for the
// reciprocal.  Prints the two distances and the CUDA error.
#include <cstdint>
#include <cstdio>

#include "rounding.cuh"

__device__ unsigned long long apart(double a, double b)
{
    const long long d = __double_as_longlong(a) - __double_as_longlong(b);
    return d < 0 ? -d : d;
}

__global__ void random_doubles(unsigned long long* most, uint64_t seed)
{
    uint64_t s = seed + (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull;
    unsigned long long r = 0, q = 0;
    for (int i = 0; i < 256; ++i) {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;                         // xorshift (Marsaglia 2003)
        const uint64_t e = 1023 - 125 + (s >> 52) % 250;
        // a quarter of the mantissas near all ones or all zeros
        uint64_t m = s & 0x000fffffffffffffull;
        if ((i & 3) == 0) m = (i & 4) ? 0x000fffffffffffffull - (m & 255) : (m & 255);
        const double x = __longlong_as_double((long long)((e << 52) | m));
        r = max(r, max(apart(sysmat::rcp64(x), 1.0 / x), apart(sysmat::rcp64(-x), 1.0 / -x)));
        q = max(q, apart(sysmat::sqrt64(x), sqrt(x)));
    }
    atomicMax(&most[0], r);
    atomicMax(&most[1], q);
}

int main()
{
    unsigned long long *most, h[2] = {99, 99};
    cudaMalloc(&most, sizeof(h));
    cudaMemset(most, 0, sizeof(h));
    for (uint64_t r = 1; r <= 4; ++r) random_doubles<<<4096, 256>>>(most, r * 0x1234567ull);
    cudaMemcpy(h, most, sizeof(h), cudaMemcpyDeviceToHost);
    std::printf("%llu %llu %d\n", h[0], h[1], (int)cudaGetLastError());
    return 0;
}
