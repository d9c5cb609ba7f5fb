// log_less (csrc/crmathf.cuh) against the double logarithm, for every word:
// prints the largest difference of the single-precision logarithm that it uses
// from the double one, and the number of words with a verdict that differs at
// one of the bounds around log u.
#include <cstdint>
#include <cstdio>

#include "crmathf.cuh"

__global__ void k_check(unsigned long long *wrong, double *worst)
{
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    const double off[] = {0.0, 1e-15, 1e-9, 1e-6, 1e-5, 0.999e-4, 0.9999e-4, 1e-4, 1.0001e-4, 1.001e-4, 2e-4, 1e-2, 1.0,
        40.0, 1e30, 1e300, inf};
    double mx = 0.0;
    unsigned long long bad = 0;
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i < 1ull << 32; i += stride) {
        const uint32_t w = static_cast<uint32_t>(i);
        const double l = ::log((static_cast<double>(w) + 0.5) * 0x1p-32);
        const float u = __fmul_rn(__fadd_rn(__uint2float_rn(w), 0.5f), 0x1p-32f);
        mx = fmax(mx, fabs(static_cast<double>(__logf(u)) - l));
        bool b = mckl_b200::log_less(w, __longlong_as_double(0x7ff8000000000000ll));  // never below a NaN
        for (double o : off) {
            const double up = l + o, dn = l - o;
            b = b || mckl_b200::log_less(w, up) != (l < up) || mckl_b200::log_less(w, dn) != (l < dn);
        }
        bad += b;
    }
    atomicAdd(wrong, bad);
    // nonnegative doubles order as integers
    atomicMax(reinterpret_cast<unsigned long long *>(worst), static_cast<unsigned long long>(__double_as_longlong(mx)));
}

int main()
{
    unsigned long long *wrong, h = 1;
    double *worst, m = 1.0;
    if (cudaMalloc(&wrong, 8) != cudaSuccess || cudaMalloc(&worst, 8) != cudaSuccess) return 1;
    cudaMemset(wrong, 0, 8);
    cudaMemset(worst, 0, 8);
    k_check<<<148 * 8, 256>>>(wrong, worst);
    if (cudaMemcpy(&h, wrong, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    if (cudaMemcpy(&m, worst, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("%llu %.6e\n", h, m);
    return 0;
}
