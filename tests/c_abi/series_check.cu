// rsqrt_series and recip_series (csrc/series.cuh) against long double and against CUDA's own
// rsqrt and division, over their whole range: prints the largest relative errors in units of
// 2^-53 and "ok", or the first value out of bounds.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "series.cuh"

__global__ void values(int n, const double *x, double *o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    o[4 * i] = cutc::rsqrt_series(x[i]);
    o[4 * i + 1] = cutc::recip_series(x[i]);
    o[4 * i + 2] = rsqrt(x[i]);
    o[4 * i + 3] = 1.0 / x[i];
}

int main()
{
    std::vector<double> x;
    uint64_t s = 88172645463325252ull;
    auto next = [&] {
        s ^= s << 13;
        s ^= s >> 7;
        return s ^= s << 17;
    };
    for (int e = -119; e < 120; e++)  // significands of all kinds in every binade
        for (int k = 0; k < 4096; k++) {
            const uint64_t r = next();
            const uint64_t m = k < 64 ? (1ull << (k % 52)) - (k / 52) : k < 128 ? ~(1ull << (k % 52)) : r;
            x.push_back(std::ldexp(1.0 + std::ldexp((double)(m & ((1ull << 52) - 1)), -52), e));
        }
    const int n = (int)x.size();
    double *dx, *dout;
    std::vector<double> o(4 * (size_t)n);
    if (cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&dout, o.size() * sizeof(double)) != cudaSuccess)
        return 2;
    cudaMemcpy(dx, x.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    values<<<(n + 255) / 256, 256>>>(n, dx, dout);
    if (cudaMemcpy(o.data(), dout, o.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 3;
    long double worst[4] = {0, 0, 0, 0};
    for (int i = 0; i < n; i++) {
        const long double ref[2] = {1.0L / std::sqrt((long double)x[i]), 1.0L / (long double)x[i]};
        for (int c = 0; c < 4; c++) {
            const long double d = c < 2 ? o[4 * i + c] - ref[c] : (long double)o[4 * i + c] - o[4 * i + c - 2];
            const long double err = std::fabs(d / ref[c & 1]) * 0x1p53L;
            worst[c] = err > worst[c] ? err : worst[c];
        }
    }
    std::printf("%d values: %.3Lf %.3Lf, against rsqrt and division %.3Lf %.3Lf\n", n, worst[0], worst[1],
                worst[2], worst[3]);
    // within 2^-52 and 2^-52.9; CUDA's rsqrt is within an ulp (2 2^-53), its division rounded
    const bool ok = worst[0] <= 2.0L && worst[1] <= 1.08L && worst[2] <= 4.0L && worst[3] <= 2.08L;
    std::puts(ok ? "ok" : "out of bounds");
    return ok ? 0 : 1;
}
