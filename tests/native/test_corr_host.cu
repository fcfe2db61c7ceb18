// Host parts of gisspa_b200/csrc/corr.cuh.
//   claims: the items of the largest launch that is allowed, and the claims behind
//   its last item, at every window
//   rings: what the autotuner tries lies around the ring that a window's rule gives
//   border: the masked indices at every window and particle diameter, to infinity
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <string>

#include "corr.cuh"

using namespace gs;

template <int N2, int V>
static int check_claims() {
    using C = CorrCfg<N2, V>;
    long long lo = 0, hi = 1ll << 31;
    while (hi - lo > 1) {
        const long long n = (lo + hi) / 2;
        (corr_units_fit(C::L, n) ? lo : hi) = n;
    }
    CorrArgs a{};
    a.nu = (int)lo;
    a.lag = 8;
    const long long items = (long long)a.nu * 2 * C::T;
    if (items >= (1ll << 31)) { printf("window %d: %lld items\n", C::L, items); return 1; }
    const int total = (int)items;
    int bad = 0;
    for (int item : {0, total / 2, total - 1}) {
        const CorrItem it = corr_item<C::T>(a, item);
        if (!corr_claimed(item, total) || it.u < 0 || it.u >= a.nu || it.j < 0 || it.j >= C::T) bad = 1;
    }
    // two claims past the end per CTA: at most 2048 threads on each of up to 256 SMs
    for (unsigned k = 0; k < 2u * 256u * (2048u / C::kThreads); ++k)
        if (corr_claimed((int)((unsigned)total + k), total)) bad = 1;
    if (bad) printf("window %d, %d vectors: claims past the last item are taken\n", C::L, V);
    return bad;
}

template <int N2>
static int check_windows() {
    if constexpr (N2 > 48) {
        return 0;
    } else {
        return check_claims<N2, 8>() | check_claims<N2, 16>() | check_windows<N2 + 1>();
    }
}

static int check_rings() {
    int bad = 0;
    for (int l = 96; l <= 752; l += 16) {
        const int tile = l <= 576 ? 8 : 16, tiles = l / tile;
        for (int threads : {512, 768, 1024}) {
            const int lag = corr_lag(148 * threads / (16 * tile), tiles), slots = (11 * lag + 4) / 5;
            const CorrRingTrials t = corr_ring_trials(slots, lag, false);
            int below = 0, above = 0, fit = 0;
            for (int s : t.slots) {
                below += s < slots && s > lag;
                above += s > slots;
                if (s < 2 || s > corr_ring_most(slots, false)) bad = 1;
            }
            for (int g : t.lags) fit += g >= 1 && g < slots && g != lag;
            if (bad || !below || !above || fit < 3) { printf("window %d: slots %d, lag %d\n", l, slots, lag); return 1; }
        }
    }
    const CorrRingTrials t = corr_ring_trials(16, 6, true);
    for (int s : t.slots) bad |= s > corr_ring_most(16, true);
    return bad;
}

static int check_border() {
    int bad = 0;
    for (int l = 96; l <= 768; l += 16)
        for (float d_m : {1e-45f, 1e-20f, 1e-5f, 1e-4f, 0.1f, 4.0f, 47.9f, 48.0f, (float)l, 1.9f * l, 2.0f * l, 2.1f * l, 3.0f * l, 4.0f * l,
                          5.0f * l, 1e6f, 8.5e9f, 9e9f, 1e20f, 3e38f, INFINITY}) {
            CorrArgs a{};
            corr_border(&a, d_m, l);
            const float q_lo = d_m / 4.0f, q_hi = (float)l - q_lo;
            for (int x = 0; x < l && !bad; ++x) {
                const int X = (x + l / 2) % l;
                const bool want = (float)X < q_lo || (float)X > q_hi;
                if (((unsigned)(x - a.yb0) <= (unsigned)(a.yb1 - a.yb0)) != want) {
                    printf("window %d, diameter %g: index %d %smasked\n", l, d_m, x, want ? "not " : "");
                    bad = 1;
                }
            }
        }
    return bad;
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int bad = 1;
    if (what == "claims") bad = check_windows<6>();
    if (what == "rings") bad = check_rings();
    if (what == "border") bad = check_border();
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
