// Compares the quotients of quotient.cuh with the division operator, bit for
// bit, on pseudorandom operands of a given kind; returns the mismatches.
#include "quotient.cuh"
#include <cmath>

namespace {
__device__ unsigned long long mix(unsigned long long x)
{
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}
// a double of random sign and mantissa, its exponent even over [lo, hi]
__device__ double any(unsigned long long h, int lo, int hi)
{
    const unsigned long long e = (unsigned long long)(lo + 1023 + (int)((h >> 52) % (unsigned)(hi - lo + 1)));
    return __longlong_as_double((long long)((h << 63) | (e << 52) | (mix(h) & 0xfffffffffffffULL)));
}
__device__ bool same(double x, double y)
{
    return __double_as_longlong(x) == __double_as_longlong(y) || (x == 0.0 && y == 0.0);
}

enum { ATANH_ARGUMENT = 0, SERIES = 1, NORMALISE = 2, MEAN_DEGREE = 3 };

__global__ void k_check(int kind, unsigned long long seed, long long n, unsigned long long* bad)
{
    unsigned long long wrong = 0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const unsigned long long h = mix(seed + (unsigned long long)q), g = mix(h ^ 0x5555);
        if (kind == ATANH_ARGUMENT) {        // (1 + x) / (1 - x), |x| < 1 down to the smallest step below 1
            double x = any(h, -60, -1);
            if (q % 3 == 0) x = copysign(1.0 - (double)(g % 4096 + 1) * 0x1p-53, x);
            const double a = __dadd_rn(1.0, x), b = __dsub_rn(1.0, x);
            wrong += !same(div_normal(a, b), __ddiv_rn(a, b));
        } else if (kind == SERIES) {         // (m - 1) / (m + 1), m in [sqrt(1/2), sqrt(2)), many next to 1
            double m = 0.70710678118654757 + 0.70710678118654757 * (double)(g >> 11) * 0x1p-53;
            if (q % 3 == 0) m = 1.0 + any(h, -52, -3);
            if (q % 1024 == 0) m = 1.0;
            const double a = __dsub_rn(m, 1.0), b = __dadd_rn(m, 1.0);
            wrong += !same(div_normal(a, b), __ddiv_rn(a, b));
        } else {                             // an entry of any exponent by its norm, or a sum by the edge count
            const double x = q % 64 == 0 ? 0.0 : any(h, -1023, 399);
            double d = kind == NORMALISE ? fabs(any(g, -200, 199)) : (double)(g % 2147483647u + 1);
            if (kind == NORMALISE && q % 5 == 0) d = __longlong_as_double(__double_as_longlong(d) | 0xfffffffffffffLL);
            const double w = __ddiv_rn(x, d);
            if (!div_by_divisor(d) || fabs(w) >= 0x1p+400 || (w != 0.0 && fabs(w) < 0x1p-1022)) continue;
            wrong += !same(div_by(x, d, 1.0 / d), w);
        }
    }
    if (wrong) atomicAdd(bad, wrong);
}
}  // namespace

// mismatches, or -1 on a CUDA error
extern "C" long long quotient_mismatches(int kind, unsigned long long seed, long long n)
{
    unsigned long long *bad = nullptr, host = 0;
    if (cudaMalloc(&bad, sizeof *bad) != cudaSuccess) return -1;
    cudaError_t e = cudaMemset(bad, 0, sizeof *bad);
    if (e == cudaSuccess) {
        k_check<<<592, 256>>>(kind, seed, n, bad);
        e = cudaMemcpy(&host, bad, sizeof host, cudaMemcpyDeviceToHost);
    }
    cudaFree(bad);
    return e == cudaSuccess ? (long long)host : -1;
}
