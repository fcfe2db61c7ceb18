// Rounding error of the specialised transforms of l = 16 N2 (k_fft16, rows) against
// that of the mixed-radix kernel on the same data, both against double.  Both take
// table entries as twiddles, the mixed-radix kernel in more stages; its error is
// the yardstick, with a quarter for the different register DFTs.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "fastfft.cuh"

using namespace gs;

static double rms(const std::vector<float2>& y, const std::vector<double2>& want) {
    double e = 0.0, t = 0.0;
    for (size_t i = 0; i < y.size(); ++i) {
        e += (y[i].x - want[i].x) * (y[i].x - want[i].x) + (y[i].y - want[i].y) * (y[i].y - want[i].y);
        t += want[i].x * want[i].x + want[i].y * want[i].y;
    }
    return sqrt(e / t);
}

template <int N2, bool kInv>
static int check() {
    using F = Fast16<N2>;
    constexpr int n = F::L, nvec = 16;
    std::mt19937 rng(N2);
    std::normal_distribution<float> nd;
    std::vector<float2> x((size_t)nvec * n), tw(n), y(x.size());
    std::vector<double2> w(n), want(x.size());
    for (auto& v : x) v = make_float2(nd(rng), nd(rng));
    for (int k = 0; k < n; ++k) {
        const double a = -2.0 * M_PI * k / n;
        tw[k] = make_float2((float)cos(a), (float)sin(a));
        w[k] = make_double2(cos(a), kInv ? -sin(a) : sin(a));
    }
    for (int v = 0; v < nvec; ++v)
        for (int k = 0; k < n; ++k) {
            double re = 0.0, im = 0.0;
            for (int m = 0; m < n; ++m) {
                const float2 a = x[(size_t)v * n + m];
                const double2 b = w[(long long)m * k % n];
                re += a.x * b.x - a.y * b.y;
                im += a.x * b.y + a.y * b.x;
            }
            want[(size_t)v * n + k] = make_double2(re, im);
        }
    float2 *dx, *dtw;
    if (cudaMalloc(&dx, 8 * x.size()) || cudaMalloc(&dtw, 8 * n)) return 1;
    cudaMemcpy(dtw, tw.data(), 8 * n, cudaMemcpyHostToDevice);
    double err[2];
    for (int which = 0; which < 2; ++which) {
        cudaMemcpy(dx, x.data(), 8 * x.size(), cudaMemcpyHostToDevice);
        if (which) {
            using IO = F16Complex<false>;
            auto kern = k_fft16<N2, kInv, false, IO>;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem_bytes());
            kern<<<dim3(nvec / F::V, 1), F::kThreads, F::smem_bytes()>>>(dtw, IO{dx, n, (long long)nvec * n, 1.0f});
        } else {
            FftDesc d{};
            d.n = n;
            d.tw = dtw;
            int m = n;
            for (int f : {8, 4, 2, 3, 5, 7, 11, 13, 17, 19, 23})
                while (m % f == 0) { d.radix[d.nst++] = f; m /= f; }
            const size_t smem = fft_smem_bytes(n, 4);
            auto kern = fft_batched_kernel<kInv, IoComplex>;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            kern<<<dim3(nvec / 4, 1), 256, smem>>>(d, VecGeom{nvec, n, 1, (long long)nvec * n}, 4, IoComplex{dx, 1.0f});
        }
        if (cudaMemcpy(y.data(), dx, 8 * y.size(), cudaMemcpyDeviceToHost) != cudaSuccess) {
            printf("%s\n", cudaGetErrorString(cudaGetLastError()));
            return 1;
        }
        err[which] = rms(y, want);
    }
    cudaFree(dx);
    cudaFree(dtw);
    if (!(err[0] < 3e-7) || !(err[1] <= 1.25 * err[0])) {
        printf("%d, inverse %d: %.3g, mixed radix %.3g\n", n, kInv, err[1], err[0]);
        return 1;
    }
    return 0;
}

int main() {
    int bad = 0;
    bad |= check<6, false>() | check<6, true>();
    bad |= check<8, false>() | check<8, true>();
    bad |= check<14, true>();
    bad |= check<19, false>();
    bad |= check<20, false>() | check<20, true>();
    bad |= check<23, true>();
    bad |= check<32, false>() | check<32, true>();
    bad |= check<45, false>() | check<45, true>();
    bad |= check<46, false>();
    bad |= check<48, false>() | check<48, true>();
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
