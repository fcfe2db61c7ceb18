// The refinement's normalised template (k_ref_norm): tm / sd within half a last
// place of double, in the given rows alone.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "refine.cuh"

using namespace gs;

int main() {
    int bad = 0;
    for (int l : {16, 96, 250}) {
        const int n = l * l, picks = 3, row0 = l / 4, row1 = l - l / 5;
        std::mt19937 rng(l);
        std::normal_distribution<float> nd;
        std::vector<float> tm((size_t)picks * n);
        for (auto& v : tm) v = nd(rng) * 0.37f;
        std::vector<RefineAcc> acc(picks);
        std::vector<double> sd(picks);
        for (int p = 0; p < picks; ++p) {
            acc[p] = RefineAcc{};
            acc[p].m1 = 0.01 * n * (p + 1);
            acc[p].m2 = p ? 0.2 * n * p : 0.0;  // the first without a positive variance: not scaled
            const double mu = acc[p].m1 / n, var = acc[p].m2 / n - mu * mu;
            sd[p] = sqrt(var > 0.0 ? var : 1.0);
        }
        char* mem = nullptr;
        const size_t bf = (size_t)picks * n * sizeof(float2), bt = (size_t)picks * n * sizeof(float);
        if (cudaMalloc(&mem, bf + bt + 4096) != cudaSuccess) return 1;
        float2* F = (float2*)mem;
        float* T = (float*)(mem + bf);
        RefineAcc* A = (RefineAcc*)(mem + (bf + bt + 7) / 8 * 8);
        cudaMemset(F, 0xff, bf);  // NaN
        cudaMemcpy(T, tm.data(), bt, cudaMemcpyHostToDevice);
        cudaMemcpy(A, acc.data(), sizeof(RefineAcc) * picks, cudaMemcpyHostToDevice);
        RefineConsts rc{};
        rc.l = l;
        rc.L2 = n;
        k_ref_norm<<<dim3(3, picks), 256>>>(T, rc, row0, row1, A, F);
        std::vector<float2> f((size_t)picks * n);
        if (cudaMemcpy(f.data(), F, bf, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        cudaFree(mem);
        double worst = 0.0;
        for (size_t i = 0; i < f.size(); ++i) {
            const int row = (int)(i % n) / l;
            if (row < row0 || row >= row1) {
                bad |= !std::isnan(f[i].x);
                continue;
            }
            const double want = (double)tm[i] / sd[i / n];
            int e;
            frexp(want, &e);
            worst = fmax(worst, fabs(f[i].x - want) / ldexp(1.0, e - 24));
            bad |= f[i].y != 0.0f;
        }
        if (bad || !(worst <= 0.5 + 1e-6)) { printf("l %d: %.4f last places\n", l, worst); bad = 1; }
    }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
