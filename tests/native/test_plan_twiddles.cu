// Twiddles of a stage of a planned transform (plan_stage): a butterfly of (1, 0, 0,
// ...) leaves the factors themselves, which have to be the table's entries, bit
// for bit, for every radix and both directions.
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

int main() {
    const int bad = check_radices<2>();
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
