// Kernels specialised for a window of l = 16 N2 pixels (N2 from 6 to 48, every
// prime factor at most 23), reached through function pointers: they are
// instantiated in winops.cu, which is compiled in parts.
#pragma once

#include "corr.cuh"

namespace gs {

struct WinOps {
    int threads_per_sm;  // of the persistent correlation, whatever the tile width
    // persistent FP32 correlation with tiles of `tile` vectors (16 or 8), at
    // most `ctas` resident CTAs per SM when ctas > 0; *fits = false (nothing
    // launched) when it does not fit on an SM
    cudaError_t (*corr)(const CorrArgs& a, int tile, int ctas, cudaStream_t st, bool* fits);
    // the same with a norm_type 1 epilogue and 16-vector tiles; nullptr for odd
    // N2 (norm_type 1 takes windows that are multiples of 32)
    cudaError_t (*corr_moments)(const CorrArgs& a, int ctas, cudaStream_t st, bool* fits);
    cudaError_t (*corr_blocks)(const CorrArgs& a, int ctas, cudaStream_t st, bool* fits);
    // forward transforms of template pairs: `tiles` tiles of 16 rows (natural or
    // PfaCols column order), and columns
    cudaError_t (*pair_rows)(const float2* tw, int nimg, int tiles, const F16PairNorm& io, cudaStream_t st);
    cudaError_t (*pair_rows_pfa)(const float2* tw, int nimg, int tiles, const F16PairNormPfa& io, cudaStream_t st);
    cudaError_t (*pair_cols)(const float2* tw, int nimg, const F16PairCols& io, cudaStream_t st);
    // forward transforms along rows of complex images, in place
    cudaError_t (*rows)(const float2* tw, int nimg, const F16Complex<false>& io, cudaStream_t st);
    // forward transform along columns, in place
    cudaError_t (*cols)(const float2* tw, int nimg, const F16Complex<true>& io, cudaStream_t st);
    // inverse transforms of the template preparation
    cudaError_t (*inv_rows)(const float2* tw, int nimg, const F16ScaleIn<false>& io, cudaStream_t st);
    cudaError_t (*inv_cols)(const float2* tw, int nimg, const F16RealOut<true>& io, cudaStream_t st);
};

// The kernels of window l, or nullptr where there are none.
const WinOps* win_ops(int l);

}  // namespace gs
