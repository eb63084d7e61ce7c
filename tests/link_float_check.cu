/* Compares the branch-free reciprocal, root and quotient of link_float.cuh with
 * the correctly rounded intrinsics; prints the number of unequal results. */
#include "link_float.cuh"

#include <cstdio>
#include <cstdlib>

__device__ unsigned long long unequal[3];

__device__ float scaled(unsigned significand, int exponent)
{
    return __uint_as_float((unsigned)(exponent + 127) << 23 | (significand & 0x7fffffu));
}

__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }

/* every significand at one exponent */
__global__ void all_significands(int exponent)
{
    const float x = scaled(blockIdx.x * blockDim.x + threadIdx.x, exponent);

    if (differ(rcp_rn(x), __frcp_rn(x)) || differ(rcp_rn(-x), __frcp_rn(-x)))
        atomicAdd(&unequal[0], 1ull);
    if (differ(sqrt_rn(x), __fsqrt_rn(x)))
        atomicAdd(&unequal[1], 1ull);
}

__device__ unsigned next(unsigned long long &s)
{
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    return (unsigned)(s >> 32);
}

/* a / b for divisors of exponent e_b and quotients of 2^-30 to 2 */
__global__ void random_quotients(int e_b, int each)
{
    unsigned long long s = (blockIdx.x * blockDim.x + threadIdx.x) * 2 + 1;
    unsigned long long bad = 0;

    s = s * 0x9E3779B97F4A7C15ull + (unsigned)(e_b + 1000);
    for (int k = 0; k < each; k++) {
        const float b = scaled(next(s), e_b);
        const float a = scaled(next(s), e_b - (int)(next(s) % 31u));

        bad += differ(div_rn(a, b, rcp_rn(b)), __fdiv_rn(a, b));
    }
    if (bad)
        atomicAdd(&unequal[2], bad);
}

int main()
{
    unsigned long long h[3] = {};

    for (int e : {-80, -79, -41, -40, -2, -1, 0, 1, 2, 39, 40, 79, 80})
        all_significands<<<1 << 13, 1 << 10>>>(e);
    for (int e = -67; e <= 67; e++)
        random_quotients<<<148 * 8, 256>>>(e, 64);
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpyFromSymbol(h, unequal, sizeof(h)) != cudaSuccess)
        return EXIT_FAILURE;
    printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return EXIT_SUCCESS;
}
