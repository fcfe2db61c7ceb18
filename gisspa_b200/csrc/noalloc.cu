// gs_correlate_window_noalloc: the correlation passes of one window without
// any device allocation.
//
// Who needs this: callers that cannot call cudaMalloc while they run, e.g.
// code inside a CUDA graph capture or an allocator-free real-time section of
// a larger pipeline, or a host that hands this library pre-allocated device
// buffers and forbids it to grow its footprint.  They keep their own input
// and output buffers; the library's intermediate maps, arg-max/sum
// accumulators and twiddle table live in one file-scope device array of fixed
// size that every GPU which loads this library holds until the process exits.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "gisspa.h"

#include "planfft.cuh"
#include "winops.hpp"

using namespace gs;

namespace {

// Fixed scratch: twiddles (first 64 KiB), accumulators (next 1 MiB), then the
// row-pass maps.  Shared by every call on a device and never cleared between
// calls except for what the call itself zeroes.
constexpr size_t kScratchBytes = GS_NOALLOC_SCRATCH_BYTES;
constexpr size_t kTwBytes = 64u << 10;
constexpr size_t kAccBytes = 1u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

// Device addresses of the scratch array, one per CUDA context.  The module
// holding the array is loaded once per context, so a context created anew
// (e.g. the primary context after cudaDeviceReset) has a new address: the
// cache is keyed by the context's unique ID, not by the device ordinal.
std::map<unsigned long long, void*> g_scratch_addr;
std::mutex g_scratch_mu;

// Unique ID of the calling thread's current context (driver API, reached
// through the runtime so that the library needs no libcuda link), or 0 when
// no context is current or the driver cannot tell.
unsigned long long current_context_id() {
    using GetCurrent = int (*)(void**);
    using GetId = int (*)(void*, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
        cudaGetLastError();
    });
    void* ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
    return id;
}

// Device address of the scratch array in the current context.  The
// host-side name g_noalloc_scratch is only a stand-in symbol, so the address
// is looked up with cudaGetSymbolAddress once per context (the first call in
// a context; that lookup also makes the device's primary context current if
// no runtime call has yet in this thread).
int scratch_for_current_device(unsigned char** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return GS_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    unsigned long long id = current_context_id();
    auto it = id ? g_scratch_addr.find(id) : g_scratch_addr.end();
    if (it != g_scratch_addr.end()) {
        *out = static_cast<unsigned char*>(it->second);
        return GS_OK;
    }
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
        cudaGetLastError();
        return GS_ERR_CUDA;
    }
    if (!id) id = current_context_id();  // the lookup may have made the context current
    if (id) g_scratch_addr[id] = p;      // without an ID nothing is cached: looked up every call
    *out = static_cast<unsigned char*>(p);
    return GS_OK;
}

// exp(-2 pi i k / n) from double-precision sincospi
__device__ __forceinline__ float2 noalloc_twiddle(int k, int n) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)n, &s, &c);
    return make_float2((float)c, (float)s);
}

// Column pass whose last CTA of an image also scores its two templates, so that
// no launch has to follow.
struct F16Pass2Last : F16Pass2 {
    int* count;    // per image, zeroed
    UnitOut* out;  // 2 per image
    __device__ void finish(double* scratch) {
        F16Pass2::finish(scratch);  // thread 0 has added the CTA's share
        if (threadIdx.x != 0) return;
        const int p = blockIdx.y;
        int prev;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(prev) : "l"(count + p) : "memory");
        if (prev != (int)gridDim.x - 1) return;
        for (int J = 2 * p; J < min(2 * p + 2, ntmpl); ++J) {
            UnitAcc a;
            a.key = __ldcg(&acc[J].key);
            a.s1 = __ldcg(&acc[J].s1);
            a.s2 = __ldcg(&acc[J].s2);
            out[J] = unit_result(a, L);
        }
    }
};

// tw[k] = exp(-2 pi i k / n) and behind them the plan's tables (plan.A = 0: none),
// zeroed accumulators and counters.
__global__ void k_noalloc_prepare(float2* tw, int n, const __grid_constant__ PlanDesc plan, UnitAcc* acc, int* count,
                                  int nacc) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nacc) {
        acc[k] = UnitAcc{0ull, 0.0, 0.0};
        count[k] = 0;
    }
    const int extra = plan.A ? plan_table_size(plan) : 0;
    if (k < n + extra) tw[k] = noalloc_twiddle(k < n ? k : plan_table_entry(plan, k - n), n);
}

// What the persistent kernel starts from: twiddles, zeroed accumulators and
// counters, the unit order (window 0, pair u).
__global__ void k_noalloc_units(float2* tw, int n, UnitAcc* acc, int2* wp, int* counters, int nu) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) tw[k] = noalloc_twiddle(k, n);
    if (k < 2 * nu) acc[k] = UnitAcc{0ull, 0.0, 0.0};
    if (k < nu) wp[k] = make_int2(0, k);
    if (k < 2 * nu + 4) counters[k] = 0;
}

int factorize_noalloc(int n, int* radix) {
    int ns = 0, m = n;
    while (m % 8 == 0 && m > 1) { radix[ns++] = 8; m /= 8; }
    while (m % 4 == 0) { radix[ns++] = 4; m /= 4; }
    while (m % 2 == 0) { radix[ns++] = 2; m /= 2; }
    for (int f : {3, 5}) while (m % f == 0) { radix[ns++] = f; m /= f; }
    for (int f = 7; (long long)f * f <= m; f += 2)
        while (m % f == 0) { radix[ns++] = f; m /= f; }
    if (m > 1) radix[ns++] = m;
    return ns;
}

template <int N2, bool kInv, bool kCols, class IO>
cudaError_t launch_fast(const float2* tw, int nimg, IO io, cudaStream_t st) {
    using F = Fast16<N2>;
    auto kern = k_fft16<N2, kInv, kCols, IO>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem_bytes());
    if (e != cudaSuccess) return e;
    kern<<<dim3(N2, nimg), F::kThreads, F::smem_bytes(), st>>>(tw, io);
    return cudaGetLastError();
}

// The planned kernel where the length has a plan and a tile fits; *done = false
// (nothing launched) otherwise.
template <bool kInv, class IO>
cudaError_t launch_plan(PlanDesc d, VecGeom g, int nimg, IO io, cudaStream_t st, bool* done) {
    *done = false;
    for (int tile = 16; d.A && tile >= 1; tile /= 2) {
        plan_layout(&d, tile);
        const size_t smem = plan_smem_bytes(d, tile);
        if (smem > (tile > 4 ? 72u << 10 : 220u << 10) || !plan_strides_fit(d, g, tile)) continue;
        auto kern = fft_plan_kernel<kInv, IO>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        if (e != cudaSuccess) return e;
        kern<<<dim3((unsigned)((g.nvec + tile - 1) / tile), nimg), 256, smem, st>>>(d, g, tile, io);
        *done = true;
        return cudaGetLastError();
    }
    return cudaSuccess;
}

template <bool kInv, class IO>
cudaError_t launch_generic(const FftDesc& d, VecGeom g, int nimg, IO io, cudaStream_t st) {
    const size_t per = 2 * (size_t)(d.n + 1) * sizeof(float2);
    size_t tile = std::max<size_t>(1, (96u << 10) / per);
    tile = std::min<size_t>(tile, 16);
    tile = std::min<size_t>(tile, (size_t)g.nvec);
    const size_t smem = fft_smem_bytes(d.n, (int)tile);
    if (smem > kMaxSmem) return cudaErrorInvalidValue;
    auto kern = fft_batched_kernel<kInv, IO>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((unsigned)((g.nvec + tile - 1) / tile), nimg), 256, smem, st>>>(d, g, (int)tile, io);
    return cudaGetLastError();
}

}  // namespace

extern "C" int gs_correlate_window_noalloc(const float* d_window_spectrum, const float* d_pair_spectra,
                                           int n_templates, int l, float d_m, gs_unit* d_units, void* stream) {
    if (!d_window_spectrum || !d_pair_spectra || !d_units || n_templates <= 0 || l < 2 || (l & 1) ||
        !(d_m > 0.0f))
        return GS_ERR_ARG;
    const size_t l2 = (size_t)l * l;
    if ((size_t)l * sizeof(float2) > kTwBytes || l2 * sizeof(float2) > kScratchBytes - kTwBytes - kAccBytes)
        return GS_ERR_UNSUPPORTED;  // beyond the fixed scratch: l <= GS_NOALLOC_MAX_WINDOW
    FftDesc desc{};
    desc.n = l;
    desc.nst = factorize_noalloc(l, desc.radix);
    if (desc.nst > kFftMaxStages) return GS_ERR_UNSUPPORTED;
    const int n2 = l / 16;
    const bool fast = l == 512 || l == 720 || l == 768;
    if (!fast && 2 * (size_t)(l + 1) * sizeof(float2) + kFftRedDoubles * sizeof(double) > kMaxSmem)
        return GS_ERR_UNSUPPORTED;
    unsigned char* base = nullptr;
    int st = scratch_for_current_device(&base);
    if (st != GS_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float2* tw = reinterpret_cast<float2*>(base);
    UnitAcc* acc = reinterpret_cast<UnitAcc*>(base + kTwBytes);
    float2* R = reinterpret_cast<float2*>(base + kTwBytes + kAccBytes);
    desc.tw = tw;
    const int npairs = (n_templates + 1) / 2;
    const size_t chunk_by_maps = (kScratchBytes - kTwBytes - kAccBytes) / (l2 * sizeof(float2));
    const size_t chunk_by_acc = kAccBytes / (2 * (sizeof(UnitAcc) + sizeof(int)));
    const int chunk = (int)std::min<size_t>(std::min(chunk_by_maps, chunk_by_acc), 65535);
    const float2* W = reinterpret_cast<const float2*>(d_window_spectrum);
    const float2* Pall = reinterpret_cast<const float2*>(d_pair_spectra);
    const float q_lo = d_m / 4.0f, q_hi = (float)l - q_lo;
    const float sgn = ((l / 2) % 2 == 0) ? 1.0f : -1.0f;

    // Windows of the persistent kernel in natural spectrum order (even N2): two
    // launches, and no map leaves L2.  The ring takes what the scratch holds.
    // Not where the two-pass kernels are specialised: a few units give the
    // persistent kernel nothing to overlap (window 512, 16 templates: 33 us
    // against 25; 768, 40 templates, whose ring has 6 slots: 171 against
    // 129); elsewhere it replaces the generic kernels (320, 20 templates: 30
    // us against 55; 736, 35: 156 against 737).
    const WinOps* ops = !fast && n2 % 2 == 0 ? win_ops(l) : nullptr;
    const int max_slots = (int)std::min<size_t>((kScratchBytes - kTwBytes - kAccBytes) / (l2 * sizeof(float2)), 1 << 20);
    if (ops && max_slots >= 4) {
        const int tile = l <= 576 ? 8 : 16, tiles = l / tile;
        int dev = 0, nsm = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return GS_ERR_CUDA;
        // per unit two accumulators, its (window, pair) and two counters
        const int per_launch = (int)((kAccBytes - 256) / (2 * sizeof(UnitAcc) + sizeof(int2) + 2 * sizeof(int)));
        const int lag0 = corr_lag(nsm * ops->threads_per_sm / (16 * tile), tiles);
        for (int p0 = 0; p0 < npairs; p0 += per_launch) {
            const int nu = std::min(per_launch, npairs - p0);
            CorrArgs a{};
            a.W = W;
            a.P = Pall + (size_t)p0 * l2;
            a.R = R;
            a.acc = acc;
            int2* wp = reinterpret_cast<int2*>(acc + 2 * (size_t)nu);
            int* counters = reinterpret_cast<int*>(wp + nu);
            a.unit_wp = wp;
            a.done_rows = counters;
            a.done_cols = counters + nu;
            a.next_item = counters + 2 * nu;
            a.error = counters + 2 * nu + 1;
            a.out = reinterpret_cast<UnitOut*>(d_units) + 2 * (size_t)p0;
            a.nu = nu;
            a.ntmpl = std::min(n_templates - 2 * p0, 2 * nu);
            a.pairs = nu;
            a.L2 = (long long)l2;
            a.S = std::min(max_slots, std::max(nu, 2));
            a.lag = nu <= max_slots ? std::min(lag0, std::min(nu, a.S - 1)) : std::max(1, std::min(lag0, 5 * a.S / 11));
            a.tw = tw;
            corr_border(&a, d_m, l);
            k_noalloc_units<<<(std::max(l, 2 * nu + 4) + 63) / 64, 64, 0, s>>>(tw, l, acc, wp, counters, nu);
            if (cudaGetLastError() != cudaSuccess) return GS_ERR_CUDA;
            bool fits = true;
            if (ops->corr(a, tile, 0, s, &fits) != cudaSuccess) return GS_ERR_CUDA;
            if (!fits) return GS_ERR_UNSUPPORTED;
        }
        return GS_OK;
    }
    PlanDesc plan;
    bool dense = false;
    if (!fast && plan_factors(l, &plan.A, &plan.B, &plan.C, &dense)) {
        plan.n = l;
        plan.dense = dense ? 1 : 0;
        plan.tw = tw;
        plan_tables(&plan, tw + l);
    } else {
        plan.A = 0;
    }
    const int ntw = l + (plan.A ? plan_table_size(plan) : 0);
    static_assert(3 * GS_NOALLOC_MAX_WINDOW * sizeof(float2) <= kTwBytes, "three tables of a window's length at most");
    for (int p0 = 0; p0 < npairs; p0 += chunk) {
        const int np = std::min(chunk, npairs - p0);
        const int nt = std::min(n_templates - 2 * p0, 2 * np);
        const float2* P = Pall + (size_t)p0 * l2;
        // accumulators start at zero for every chunk
        int* count = reinterpret_cast<int*>(acc + 2 * (size_t)np);
        k_noalloc_prepare<<<(std::max(ntw, 2 * np) + 63) / 64, 64, 0, s>>>(tw, l, plan, acc, count, 2 * np);
        if (cudaGetLastError() != cudaSuccess) return GS_ERR_CUDA;
        cudaError_t e;
        if (fast) {
            F16Pass1 io1{W, P, R, l, (long long)l2};
            F16Pass2Last io2;
            io2.R = R; io2.acc = acc; io2.L = l; io2.ntmpl = nt; io2.L2 = (long long)l2;
            io2.q_lo = q_lo; io2.q_hi = q_hi; io2.sgn = sgn;
            io2.count = count;
            io2.out = reinterpret_cast<UnitOut*>(d_units) + 2 * (size_t)p0;
            switch (n2) {
                case 32: e = launch_fast<32, true, false>(tw, np, io1, s);
                         if (e == cudaSuccess) e = launch_fast<32, true, true>(tw, np, io2, s); break;
                case 45: e = launch_fast<45, true, false>(tw, np, io1, s);
                         if (e == cudaSuccess) e = launch_fast<45, true, true>(tw, np, io2, s); break;
                default: e = launch_fast<48, true, false>(tw, np, io1, s);
                         if (e == cudaSuccess) e = launch_fast<48, true, true>(tw, np, io2, s); break;
            }
            if (e != cudaSuccess) return GS_ERR_CUDA;
            continue;
        } else {
            const VecGeom rows{l, (long long)l, 1, (long long)l2};
            const VecGeom cols{l, 1, (long long)l, (long long)l2};
            IoPass1 io1{W, P, R, (long long)l2};
            IoPass2 io2;
            io2.R = R; io2.acc = acc; io2.l = l; io2.ntmpl = nt; io2.q_lo = q_lo; io2.q_hi = q_hi; io2.sgn = sgn;
            bool done = false;
            e = launch_plan<true>(plan, rows, np, io1, s, &done);
            if (e == cudaSuccess && !done) e = launch_generic<true>(desc, rows, np, io1, s);
            if (e == cudaSuccess) e = launch_plan<true>(plan, cols, np, io2, s, &done);
            if (e == cudaSuccess && !done) e = launch_generic<true>(desc, cols, np, io2, s);
        }
        if (e != cudaSuccess) return GS_ERR_CUDA;
        k_finalize<<<(nt + 127) / 128, 128, 0, s>>>(acc, nt, l, reinterpret_cast<UnitOut*>(d_units) + 2 * (size_t)p0);
        if (cudaGetLastError() != cudaSuccess) return GS_ERR_CUDA;
    }
    return GS_OK;
}
