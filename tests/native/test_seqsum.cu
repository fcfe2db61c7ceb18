// The running sums of gisspa_b200/csrc/seqsum.cuh against a plain loop of
// float additions, bit for bit: runs of 16 terms composed in a tree and
// applied or added term by term (on the CPU, without arguments), and the
// kernel (with the argument "gpu").  The terms cover ties in both parities,
// stalls, binade changes, sums around zero, and values that must not be
// applied as a run.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <string>
#include <vector>

#include "seqsum.cuh"

using namespace gs;

static float plain(const std::vector<float>& q) {
    volatile float s = 0.0f;
    for (float v : q) s = s + v;
    return s;
}

static bool same(float a, float b) { return (a != a && b != b) || seq_bits(a) == seq_bits(b); }

// 512 terms at a time, as one warp's unit
static float by_runs(const std::vector<float>& q, long long* applied) {
    float s = 0.0f;
    for (size_t b = 0; b < q.size(); b += 512) {
        const unsigned binade = seq_binade(s);
        SeqRun lane[32];
        for (int c = 0; c < 32; ++c) {
            float t[16];
            for (int i = 0; i < 16; ++i) t[i] = b + c * 16 + i < q.size() ? q[b + c * 16 + i] : 0.0f;
            lane[c] = binade ? seq_run(t, seq_scale(binade)) : seq_identity();
        }
        for (int off = 1; off < 32; off *= 2)
            for (int c = 0; c + off < 32; c += 2 * off) lane[c] = seq_then(lane[c], lane[c + off]);
        if (seq_apply(s, binade, lane[0])) {
            ++*applied;
        } else {
            volatile float v = s;
            for (size_t i = b; i < q.size() && i < b + 512; ++i) v = v + q[i];
            s = v;
        }
    }
    return s;
}

static std::vector<std::vector<float>> cases() {
    std::vector<std::vector<float>> out;
    std::mt19937 rng(7);
    std::normal_distribution<float> gauss;
    std::uniform_real_distribution<float> uni;
    auto add = [&](size_t n, auto f) {
        std::vector<float> q(n);
        for (size_t i = 0; i < n; ++i) q[i] = f(i);
        out.push_back(q);
    };
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    for (size_t n : {1ul, 15ul, 511ul, 16384ul, 16385ul, 100003ul, 400000ul}) {
        const float inv = 1.0f / (float)n;
        add(n, [&](size_t) { return gauss(rng) * inv; });                             // around zero
        add(n, [&](size_t) { const float v = gauss(rng); return v * v * inv; });      // rising, stalls
        add(n, [&](size_t) { return (12.0f + 3.0f * gauss(rng)) * inv; });
        add(n, [&](size_t) { return -(1.0f + uni(rng)) * inv; });                     // negative
        add(n, [&](size_t) { return std::ldexp((float)(int)(rng() % 9), -24); });     // halves of the last place
        add(n, [&](size_t i) { return i == 0 ? 1.0f : std::ldexp(1.0f + (rng() & 1), -24); });
        add(n, [&](size_t i) { return i == 0 ? -3.0f : std::ldexp((float)((int)(rng() % 5) - 2), -23); });
        add(n, [&](size_t i) { return i % 1000 == 999 ? 2.0f * gauss(rng) : 1e-6f * gauss(rng); });
        add(n, [&](size_t) { return 0.0f; });
        add(n, [&](size_t i) { return i < n / 2 ? inv : -inv; });                     // up and back
        add(n, [&](size_t) { return 1e-38f * uni(rng); });
        add(n, [&](size_t) { return 3e37f * uni(rng); });
        add(n, [&](size_t i) { return i == n / 2 ? nan : inv; });
        add(n, [&](size_t i) { return i == n / 3 ? inf : inv; });
    }
    return out;
}

int main(int argc, char** argv) {
    const bool gpu = argc > 1 && std::string(argv[1]) == "gpu";
    const auto cs = cases();
    int bad = 0;
    long long applied = 0;
    for (size_t c = 0; c < cs.size(); ++c) {
        const float want = plain(cs[c]);
        if (!gpu) {
            const float got = by_runs(cs[c], &applied);
            if (!same(got, want)) { printf("case %zu (n %zu): %.9g, plain %.9g\n", c, cs[c].size(), got, want); bad = 1; }
            continue;
        }
        // both arrays of one launch: this case and the next one cut or padded to its length
        const size_t n = cs[c].size(), n4 = (n + 3) / 4 * 4;
        std::vector<float> two(2 * n4, 0.0f), other(cs[(c + 1) % cs.size()]);
        other.resize(n, 0.0f);
        memcpy(two.data(), cs[c].data(), 4 * n);
        memcpy(two.data() + n4, other.data(), 4 * n);
        const int nblk = (int)((n + kSeqBlock - 1) / kSeqBlock);
        std::vector<double> exact(2 * nblk, 0.0);
        for (size_t i = 0; i < n; ++i) {
            exact[i / kSeqBlock] += two[i];
            exact[nblk + i / kSeqBlock] += two[n4 + i];
        }
        // the second time with predictions that are no good: only the route may change
        for (int bad_guess = 0; bad_guess < 2; ++bad_guess) {
            if (bad_guess)
                for (double& e : exact) e *= 0.37;
            float *d = nullptr, *ds = nullptr, got[2] = {0, 0};
            double* de = nullptr;
            SeqBlock* db = nullptr;
            if (cudaMalloc(&d, 8 * n4) || cudaMalloc(&ds, 8) || cudaMalloc(&de, 16 * nblk) ||
                cudaMalloc(&db, 2 * nblk * sizeof(SeqBlock)))
                return 2;
            cudaMemcpy(d, two.data(), 8 * n4, cudaMemcpyHostToDevice);
            cudaMemcpy(de, exact.data(), 16 * nblk, cudaMemcpyHostToDevice);
            cudaFuncSetAttribute(k_seq_apply, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSeqSmem);
            k_seq_runs<<<dim3(nblk, 2), kSeqThreads>>>(d, (long long)n4, (long long)n, de, db);
            k_seq_apply<<<2, kSeqThreads, kSeqSmem>>>(d, (long long)n4, (long long)n, db, nblk, ds);
            if (cudaMemcpy(got, ds, 8, cudaMemcpyDeviceToHost) != cudaSuccess) { printf("%s\n", cudaGetErrorString(cudaGetLastError())); return 2; }
            cudaFree(d);
            cudaFree(ds);
            cudaFree(de);
            cudaFree(db);
            const float want2 = plain(other);
            if (!same(got[0], want) || !same(got[1], want2)) {
                printf("case %zu (n %zu): %.9g %.9g, plain %.9g %.9g\n", c, n, got[0], got[1], want, want2);
                bad = 1;
            }
        }
    }
    if (!gpu && applied < 1000) { printf("only %lld runs applied\n", applied); bad = 1; }
    if (!bad) printf("OK\n");
    return bad;
}
