// A dependency wait of the persistent correlation that runs out (its counter
// starts one short, so the tiles of unit 1 that it stands for never reach the
// target): the launch ends, raises its flag and scores that unit NaN; the units
// before it, and the same launch with whole counters, score as they should.  (CTAs
// that wait hold items of later units, whose waits may give up as well.)
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "corr.cuh"

using namespace gs;

int main() {
    constexpr int N2 = 6, V = 8, L = 16 * N2, nu = 4;
    using C = CorrCfg<N2, V>;
    const long long l2 = (long long)L * L;
    std::mt19937 rng(1);
    std::normal_distribution<float> nd;
    std::vector<float2> w(l2), p(nu * l2), tw(L);
    for (auto& v : w) v = make_float2(nd(rng), nd(rng));
    for (auto& v : p) v = make_float2(nd(rng), nd(rng));
    for (int k = 0; k < L; ++k) tw[k] = make_float2((float)cos(-2 * M_PI * k / L), (float)sin(-2 * M_PI * k / L));
    std::vector<int2> wp(nu);
    for (int u = 0; u < nu; ++u) wp[u] = make_int2(0, u);
    char* mem = nullptr;
    const size_t bw = sizeof(float2) * l2;
    if (cudaMalloc(&mem, (1 + 2 * nu) * bw + (1 << 16)) != cudaSuccess) return 1;
    CorrArgs a{};
    float2* W = (float2*)mem;
    float2* P = W + l2;
    a.W = W; a.P = P; a.R = P + nu * l2;
    char* rest = mem + (1 + 2 * nu) * bw;
    float2* dtw = (float2*)rest;
    int2* dwp = (int2*)(rest + 8 * L);
    a.acc = (UnitAcc*)(rest + 4096);
    a.out = (UnitOut*)(rest + 8192);
    int* cnt = (int*)(rest + 12288);
    a.tw = dtw; a.unit_wp = dwp;
    a.done_rows = cnt; a.done_cols = cnt + nu; a.next_item = cnt + 2 * nu; a.error = cnt + 2 * nu + 1;
    a.nu = nu; a.ntmpl = 2 * nu; a.pairs = nu; a.S = nu; a.lag = 1; a.L2 = l2;
    corr_border(&a, 20.0f, L);
    cudaMemcpy(W, w.data(), bw, cudaMemcpyHostToDevice);
    cudaMemcpy(P, p.data(), nu * bw, cudaMemcpyHostToDevice);
    cudaMemcpy(dtw, tw.data(), 8 * L, cudaMemcpyHostToDevice);
    cudaMemcpy(dwp, wp.data(), sizeof(int2) * nu, cudaMemcpyHostToDevice);
    std::vector<UnitOut> out[2];
    int flag[2];
    for (int t = 0; t < 2; ++t) {
        std::vector<int> c(2 * nu + 4, 0);
        if (t) c[1] = -1;  // unit 1's rows
        cudaMemset(a.acc, 0, sizeof(UnitAcc) * 2 * nu);
        cudaMemset(a.out, 0, sizeof(UnitOut) * 2 * nu);
        cudaMemcpy(cnt, c.data(), sizeof(int) * c.size(), cudaMemcpyHostToDevice);
        k_corr_persistent<N2, V><<<64, C::kThreads, CorrSmem<N2, V>::bytes>>>(a);
        out[t].resize(2 * nu);
        if (cudaMemcpy(out[t].data(), a.out, sizeof(UnitOut) * 2 * nu, cudaMemcpyDeviceToHost) != cudaSuccess) {
            printf("%s\n", cudaGetErrorString(cudaGetLastError()));
            return 1;
        }
        cudaMemcpy(&flag[t], a.error, sizeof(int), cudaMemcpyDeviceToHost);
    }
    int bad = 0;
    if (flag[0] || !flag[1]) { printf("flags %d %d\n", flag[0], flag[1]); bad = 1; }
    for (int J = 0; J < 2 * nu; ++J) {
        const float good = out[0][J].score, late = out[1][J].score;
        if (!(good > 1.0f)) { printf("template %d: %g\n", J, good); bad = 1; }
        // sums of squares are added in any order
        const bool same = std::fabs(late - good) <= 1e-6f * good;
        const bool waited = J / 2 == 1;
        if (waited ? !std::isnan(late) : J < 2 ? !same : !(std::isnan(late) || same)) {
            printf("template %d after the wait gave up: %g (%g)\n", J, late, good);
            bad = 1;
        }
    }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
