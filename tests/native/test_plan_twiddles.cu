// Twiddles of a stage of a planned transform (plan_stage): a butterfly of (1, 0, 0,
// ...) leaves the factors themselves, which have to be the table's entries, bit
// for bit, for every radix and both directions; and a transform with the stages' own
// tables (plan_tables) is the one without them bit for bit, columns and rows.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "planfft.cuh"

using namespace gs;

template <int R, bool kInv>
__global__ void k_stage(const float2* tw, int m, float2* out) {
    extern __shared__ float2 buf[];
    for (int i = threadIdx.x; i < R * m; i += blockDim.x) buf[i] = make_float2(i < m ? 1.0f : 0.0f, 0.0f);
    __syncthreads();
    // one vector, m butterflies j with entries j + m q, factors W_n^{q j}, n = R m
    const PlanStage s{SmallDiv{(unsigned)m, (unsigned)(((1ull << 32) + m - 1) / m)},
                      SmallDiv{(unsigned)m, (unsigned)(((1ull << 32) + m - 1) / m)}, 0, 1, m, 1, false};
    plan_stage<R, kInv, true>(buf, 1, R * m, s, tw);
    for (int i = threadIdx.x; i < R * m; i += blockDim.x) out[i] = buf[i];
}

template <int R, bool kInv>
static int check() {
    const int m = 97, n = R * m;
    std::vector<float2> tw(n), y(n);
    for (int k = 0; k < n; ++k) tw[k] = make_float2((float)cos(-2 * M_PI * k / n), (float)sin(-2 * M_PI * k / n));
    float2 *dtw, *dy;
    if (cudaMalloc(&dtw, 8 * n) || cudaMalloc(&dy, 8 * n)) return 1;
    cudaMemcpy(dtw, tw.data(), 8 * n, cudaMemcpyHostToDevice);
    k_stage<R, kInv><<<1, 256, 8 * n>>>(dtw, m, dy);
    if (cudaMemcpy(y.data(), dy, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    cudaFree(dtw);
    cudaFree(dy);
    int wrong = 0;
    for (int q = 0; q < R; ++q)
        for (int j = 0; j < m; ++j) {
            const float2 w = tw[q * j], a = y[q * m + j];
            wrong += a.x != w.x || a.y != (kInv ? -w.y : w.y);
        }
    if (wrong) printf("radix %d, inverse %d: %d of %d factors differ\n", R, kInv, wrong, n);
    return wrong != 0;
}

template <int R>
static int check_radices() {
    if constexpr (R > 23) {
        return 0;
    } else {
        int bad = 0;
        if constexpr (plan_radix(R) && R > 1) bad = check<R, false>() | check<R, true>();
        return bad | check_radices<R + 1>();
    }
}

template <bool kInv>
static int check_tables(int n, bool cols) {
    const int nvec = 5, tile = 4;
    PlanDesc d;
    bool dense = false;
    if (!plan_factors(n, &d.A, &d.B, &d.C, &dense)) { printf("no plan for %d\n", n); return 1; }
    d.n = n;
    d.dense = dense;
    plan_layout(&d, tile);
    const size_t smem = plan_smem_bytes(d, tile);
    if (smem > kMaxSmem) return 0;  // such a tile is not launched
    std::vector<float2> tw(n), x((size_t)nvec * n), y[2];
    for (int k = 0; k < n; ++k) tw[k] = make_float2((float)cos(-2 * M_PI * k / n), (float)sin(-2 * M_PI * k / n));
    const int extra = plan_table_size(d);
    for (int i = 0; i < extra; ++i) {
        const int k = plan_table_entry(d, i);
        if (k < 0 || k >= n) { printf("n %d: entry %d is %d\n", n, i, k); return 1; }
        tw.push_back(tw[k]);
    }
    for (size_t i = 0; i < x.size(); ++i) x[i] = make_float2(sinf(0.37f * i), cosf(1.1f * (i % 1009)));
    float2 *dx, *dtw;
    if (cudaMalloc(&dx, 8 * x.size()) || cudaMalloc(&dtw, 8 * tw.size())) return 1;
    cudaMemcpy(dtw, tw.data(), 8 * tw.size(), cudaMemcpyHostToDevice);
    d.tw = dtw;
    const VecGeom g = cols ? VecGeom{nvec, 1, nvec, (long long)nvec * n} : VecGeom{nvec, n, 1, (long long)nvec * n};
    auto kern = fft_plan_kernel<kInv, IoComplex>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    for (int t = 0; t < 2; ++t) {
        if (t) plan_tables(&d, dtw + n);
        cudaMemcpy(dx, x.data(), 8 * x.size(), cudaMemcpyHostToDevice);
        kern<<<dim3((nvec + tile - 1) / tile, 1), 256, smem>>>(d, g, tile, IoComplex{dx, 1.0f});
        y[t].resize(x.size());
        if (cudaMemcpy(y[t].data(), dx, 8 * x.size(), cudaMemcpyDeviceToHost) != cudaSuccess) {
            printf("%s\n", cudaGetErrorString(cudaGetLastError()));
            return 1;
        }
    }
    cudaFree(dx);
    cudaFree(dtw);
    if (memcmp(y[0].data(), y[1].data(), 8 * x.size())) {
        printf("n %d (%d x %d x %d): tables differ\n", n, d.A, d.B, d.C);
        return 1;
    }
    return 0;
}

int main() {
    int bad = check_radices<2>();
    for (int n : {7, 29, 36, 58, 300, 341, 512, 1190, 1443, 4096, 5760})
        for (int cols = 0; cols < 2; ++cols) bad |= check_tables<false>(n, cols) | check_tables<true>(n, cols);
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
