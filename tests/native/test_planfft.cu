// gisspa_b200/csrc/planfft.cuh: the factor plans of every length up to 6000
// (on the CPU, without arguments), and the kernel with the argument "gpu":
// rows and columns of a ragged number of vectors, both directions, against a
// double-precision DFT of a few outputs of every vector.
#include <cmath>
#include <cstdio>
#include <random>
#include <string>
#include <vector>

#include "planfft.cuh"

using namespace gs;

static int check_plans() {
    int bad = 0, none = 0;
    for (int n = 2; n <= 6000; ++n) {
        int A = 0, B = 0, C = 0;
        bool dense = false;
        if (!plan_factors(n, &A, &B, &C, &dense)) { ++none; continue; }
        if ((long long)A * B * C != n || !plan_radix(A) || !plan_radix(B) || (!dense && !plan_radix(C)) ||
            (dense && (C > kPlanMaxPrime || C % 2 == 0))) {
            printf("n %d: %d x %d x %d\n", n, A, B, C);
            bad = 1;
        }
    }
    // the detectors' sides, the windows and their likes have one
    for (int n : {3838, 3710, 4096, 5760, 4092, 1024, 512, 300, 320, 720, 768, 1443, 1190}) {
        int A, B, C;
        bool dense;
        if (!plan_factors(n, &A, &B, &C, &dense)) { printf("no plan for %d\n", n); bad = 1; }
    }
    printf("%d lengths without a plan\n", none);
    return bad;
}

template <bool kInv>
static int check_gpu(int n, int nvec, bool cols, int tile) {
    PlanDesc d;
    bool dense = false;
    if (!plan_factors(n, &d.A, &d.B, &d.C, &dense)) { printf("no plan for %d\n", n); return 1; }
    d.n = n;
    d.dense = dense;
    plan_layout(&d, tile);
    const size_t smem = plan_smem_bytes(d, tile);
    if (smem > 227 * 1024) return 0;  // such a tile is not launched
    std::mt19937 rng(n);
    std::normal_distribution<float> nd;
    const int img = 2;
    std::vector<float2> x((size_t)img * nvec * n), y(x.size()), tw(n);
    for (auto& v : x) v = make_float2(nd(rng), nd(rng));
    for (int k = 0; k < n; ++k) tw[k] = make_float2((float)cos(-2 * M_PI * k / n), (float)sin(-2 * M_PI * k / n));
    float2 *dx, *dtw;
    if (cudaMalloc(&dx, 8 * x.size()) || cudaMalloc(&dtw, 8 * n)) return 1;
    cudaMemcpy(dx, x.data(), 8 * x.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(dtw, tw.data(), 8 * n, cudaMemcpyHostToDevice);
    d.tw = dtw;
    const VecGeom g = cols ? VecGeom{nvec, 1, nvec, (long long)nvec * n} : VecGeom{nvec, n, 1, (long long)nvec * n};
    auto kern = fft_plan_kernel<kInv, IoComplex>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<dim3((nvec + tile - 1) / tile, img), 256, smem>>>(d, g, tile, IoComplex{dx, 1.0f});
    if (cudaMemcpy(y.data(), dx, 8 * y.size(), cudaMemcpyDeviceToHost) != cudaSuccess) { printf("%s\n", cudaGetErrorString(cudaGetLastError())); return 1; }
    cudaFree(dx);
    cudaFree(dtw);
    double err = 0, top = 0;
    for (int i = 0; i < img; ++i)
        for (int v = 0; v < nvec; ++v)
            for (int c = 0; c < 24; ++c) {
                const int k = c < 12 ? (int)((long long)c * (n - 1) / 11) : (int)(rng() % n);
                double sr = 0, si = 0;
                for (int m = 0; m < n; ++m) {
                    const float2 a = x[vec_addr(g, i, v, m)];
                    const double w = (kInv ? 2 : -2) * M_PI * ((long long)m * k % n) / n;
                    sr += a.x * cos(w) - a.y * sin(w);
                    si += a.x * sin(w) + a.y * cos(w);
                }
                const float2 b = y[vec_addr(g, i, v, k)];
                err = fmax(err, hypot(b.x - sr, b.y - si));
                top = fmax(top, hypot(sr, si));
            }
    if (!(err <= 2e-6 * top)) { printf("n %d (%d x %d x %d) cols %d tile %d inv %d: %.3g\n", n, d.A, d.B, d.C, cols, tile, kInv, err / top); return 1; }
    return 0;
}

int main(int argc, char** argv) {
    int bad = check_plans();
    if (argc > 1 && std::string(argv[1]) == "gpu")
        for (int n : {2, 7, 19, 23, 29, 36, 58, 97, 250, 300, 341, 512, 607, 720, 988, 1021, 1190, 1443, 3710, 3838, 4092, 4096, 5760})
            for (int tile : {1, 2, 4, 8, 16})
                for (int cols = 0; cols < 2; ++cols) {
                    const int nvec = n > 1000 ? tile + 1 : 2 * tile + 3;
                    bad |= check_gpu<false>(n, nvec, cols, tile);
                    bad |= check_gpu<true>(n, nvec, cols, tile);
                }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
