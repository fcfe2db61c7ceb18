// Host parts of gisspa_b200/csrc/corr.cuh.
//   claims: the items of the largest launch that is allowed, and the claims behind
//   its last item, at every window
#include <cstdio>
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

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int bad = 1;
    if (what == "claims") bad = check_windows<6>();
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
