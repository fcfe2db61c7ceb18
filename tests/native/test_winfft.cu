// Host-side check of the transforms behind the windows l = 16 N2
// (gisspa_b200/csrc/winops.hpp): the register DFT of every length N2 from 6 to
// 48 that has one, both directions, and for odd N2 the prime-factor maps of
// the correlation, against a double-precision DFT.  Built with nvcc and run on
// the CPU by tests/test_native_windows.py.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "corr.cuh"

using namespace gs;

static std::mt19937 rng(5);

template <int N, bool kInv>
static double dft_error() {
    std::normal_distribution<double> nd;
    float2 x[N], a[N];
    for (int n = 0; n < N; ++n) a[n] = x[n] = make_float2((float)nd(rng), (float)nd(rng));
    rf::rfft<N, 1, kInv>(a);
    double err = 0, top = 0;
    for (int k = 0; k < N; ++k) {
        double sr = 0, si = 0;
        for (int n = 0; n < N; ++n) {
            const double w = (kInv ? 2.0 : -2.0) * M_PI * (n * k % N) / N;
            sr += x[n].x * cos(w) - x[n].y * sin(w);
            si += x[n].x * sin(w) + x[n].y * cos(w);
        }
        const float2 g = a[rf::rpos<N>(k)];
        err = fmax(err, hypot(g.x - sr, g.y - si));
        top = fmax(top, hypot(sr, si));
    }
    return err / top;
}

// one inverse transform of length 16 N2 the correlation's way
template <int N2>
static double window_error() {
    using F = CorrCfg<N2, 8>;
    constexpr int L = 16 * N2;
    std::normal_distribution<double> nd;
    std::vector<float2> spec(L), in(L), out(L);
    for (int k = 0; k < L; ++k) spec[k] = make_float2((float)nd(rng), (float)nd(rng));
    // odd N2: the spectrum is read in the prime-factor order; even N2: natural order and twiddles
    for (int p = 0; p < L; ++p) in[p] = spec[F::spectrum_row(p)];
    if (F::kPfa) {
        const PfaCols pc = PfaCols::make(L);
        for (int p = 0; p < L; ++p)
            if (pc.logical(p) != F::spectrum_row(p) || pc.physical(pc.logical(p)) != p) return 1.0;
    }
    std::vector<float2> mid(L);
    for (int n2 = 0; n2 < N2; ++n2) {
        float2 x[16];
        for (int n1 = 0; n1 < 16; ++n1) x[n1] = in[n2 + N2 * n1];
        rf::rfft<16, 1, true>(x);
        for (int k1 = 0; k1 < 16; ++k1) {
            float2 v = x[rf::rpos<16>(k1)];
            if (!F::kPfa) {
                const double w = 2.0 * M_PI * (n2 * k1 % L) / L;
                v = cmul(v, make_float2((float)cos(w), (float)sin(w)));
            }
            mid[k1 * N2 + n2] = v;
        }
    }
    for (int k1 = 0; k1 < 16; ++k1) {
        float2 b[N2];
        for (int n2 = 0; n2 < N2; ++n2) b[n2] = mid[k1 * N2 + n2];
        rf::rfft<N2, 1, true>(b);
        for (int k2 = 0; k2 < N2; ++k2) out[F::kPfa ? F::map_coord(k1, k2) : k1 + 16 * k2] = b[rf::rpos<N2>(k2)];
    }
    double err = 0, top = 0;
    for (int x = 0; x < L; ++x) {
        double sr = 0, si = 0;
        for (int k = 0; k < L; ++k) {
            const double w = 2.0 * M_PI * ((long long)x * k % L) / L;
            sr += spec[k].x * cos(w) - spec[k].y * sin(w);
            si += spec[k].x * sin(w) + spec[k].y * cos(w);
        }
        err = fmax(err, hypot(out[x].x - sr, out[x].y - si));
        top = fmax(top, hypot(sr, si));
    }
    return err / top;
}

template <int N2>
static int check() {
    int bad = 0;
    if constexpr (N2 <= 48) {
        if constexpr (rf::rfft_exists(N2)) {
            const double e = fmax(fmax(dft_error<N2, false>(), dft_error<N2, true>()), window_error<N2>());
            if (!(e < 2e-6)) { printf("N2 %d: %.3g\n", N2, e); bad = 1; }
        }
        bad |= check<N2 + 1>();
    }
    return bad;
}

int main() {
    const int bad = check<6>();
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
