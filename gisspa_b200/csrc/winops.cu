// Instantiations of winops.hpp.  Compiled GS_WIN_PARTS times, part GS_WIN_PART
// holding the windows with N2 % GS_WIN_PARTS == GS_WIN_PART (each N2 takes
// ptxas several seconds).
#include "winops.hpp"

#ifndef GS_WIN_PARTS
#error "GS_WIN_PARTS and GS_WIN_PART are set by the build"
#endif

namespace gs {

namespace {

template <int N2, bool kInv, bool kCols, class IO>
cudaError_t fft_launch_tiles(const float2* tw, int nimg, int tiles, const IO& io, cudaStream_t st) {
    using F = Fast16<N2>;
    auto kern = k_fft16<N2, kInv, kCols, IO>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem_bytes());
    if (e != cudaSuccess) return e;
    kern<<<dim3((unsigned)tiles, (unsigned)nimg), F::kThreads, F::smem_bytes(), st>>>(tw, io);
    return cudaGetLastError();
}

template <int N2, bool kInv, bool kCols, class IO>
cudaError_t fft_launch(const float2* tw, int nimg, const IO& io, cudaStream_t st) {
    return fft_launch_tiles<N2, kInv, kCols>(tw, nimg, N2, io, st);
}

template <int N2, int V, CorrEpi kEpi = kCorrScore>
cudaError_t corr_launch_v(const CorrArgs& a, int ctas, cudaStream_t st, bool* fits) {
    using C = CorrCfg<N2, V>;
    constexpr size_t smem = CorrSmem<N2, V>::bytes;
    auto kern = k_corr_persistent<N2, V, kEpi>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0, nsm = 0, dev = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::kThreads, smem);
    if (e != cudaSuccess) return e;
    *fits = per_sm >= 1;
    if (!*fits) return cudaSuccess;
    if (ctas > 0 && ctas < per_sm) per_sm = ctas;
    const long long items = (long long)a.nu * 2 * C::T;
    const long long grid = (long long)nsm * per_sm < items ? (long long)nsm * per_sm : items;
    kern<<<(unsigned)grid, C::kThreads, smem, st>>>(a);
    return cudaGetLastError();
}

template <int N2>
cudaError_t corr_launch(const CorrArgs& a, int tile, int ctas, cudaStream_t st, bool* fits) {
    return tile == 8 ? corr_launch_v<N2, 8>(a, ctas, st, fits) : corr_launch_v<N2, 16>(a, ctas, st, fits);
}

template <int N2>
struct Ops {
    static constexpr bool kHere = rf::rfft_exists(N2) && N2 % GS_WIN_PARTS == GS_WIN_PART;
    static const WinOps* get() {
        if constexpr (kHere) {
            static const WinOps ops = [] {
                WinOps o{};
                o.threads_per_sm = CorrCfg<N2, 16>::kThreadsPerSm;
                o.corr = corr_launch<N2>;
                if constexpr (N2 % 2 == 0) {
                    o.corr_moments = corr_launch_v<N2, 16, kCorrMoments>;
                    o.corr_blocks = corr_launch_v<N2, 16, kCorrBlocks>;
                }
                if constexpr (N2 % 2 == 1) o.pair_rows_pfa = fft_launch_tiles<N2, false, false, F16PairNormPfa>;
                o.pair_rows = fft_launch_tiles<N2, false, false, F16PairNorm>;
                o.pair_cols = fft_launch<N2, false, true, F16PairCols>;
                o.rows = fft_launch<N2, false, false, F16Complex<false>>;
                o.cols = fft_launch<N2, false, true, F16Complex<true>>;
                o.inv_rows = fft_launch<N2, true, false, F16ScaleIn<false>>;
                o.inv_cols = fft_launch<N2, true, true, F16RealOut<true>>;
                return o;
            }();
            return &ops;
        } else {
            return nullptr;
        }
    }
};

template <int N2>
const WinOps* find(int n2) {
    if constexpr (N2 > 48) {
        return nullptr;
    } else {
        return n2 == N2 ? Ops<N2>::get() : find<N2 + 1>(n2);
    }
}

}  // namespace

#define GS_CAT2(a, b) a##b
#define GS_CAT(a, b) GS_CAT2(a, b)
const WinOps* GS_CAT(win_ops_part, GS_WIN_PART)(int n2) { return find<6>(n2); }

}  // namespace gs
