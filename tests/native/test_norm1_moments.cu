// k_norm1_moments2: the reciprocal deviation is the correctly rounded one of the
// float variance (half a last place, against double), 0 and -1 where it has to be.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "norm1.cuh"

using namespace gs;

int main() {
    const int n = 1 << 20;
    const float total = 12.0f;
    std::mt19937 rng(3);
    std::uniform_real_distribution<float> e(-80.0f, 80.0f);
    std::vector<float2> s(n), r(n);
    // means of 0, so that the variance is one division
    for (auto& v : s) v = make_float2(0.0f, exp2f(e(rng)));
    s[0].y = 0.0f;
    s[1].y = -1.0f;
    s[2].y = INFINITY;
    s[3].y = NAN;
    s[4] = make_float2(NAN, 1.0f);
    float2* d;
    if (cudaMalloc(&d, 8 * n) != cudaSuccess) return 1;
    cudaMemcpy(d, s.data(), 8 * n, cudaMemcpyHostToDevice);
    k_norm1_moments2<<<(n + 255) / 256, 256>>>(d, n, total);
    if (cudaMemcpy(r.data(), d, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    int bad = 0;
    const float special[5] = {-1.0f, -1.0f, 0.0f, -1.0f, -1.0f};
    for (int i = 0; i < 5; ++i)
        if (r[i].y != special[i]) { printf("%g: %g\n", s[i].y, r[i].y); bad = 1; }
    double worst = 0.0;
    for (int i = 5; i < n; ++i) {
        const double want = 1.0 / sqrt((double)(s[i].y / total));
        int ex;
        frexp(want, &ex);
        worst = fmax(worst, fabs(r[i].y - want) / ldexp(1.0, ex - 24));
    }
    // double rounding adds nothing that shows beside half a place
    if (!(worst <= 0.5 + 1e-6)) { printf("%.4f last places\n", worst); bad = 1; }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
