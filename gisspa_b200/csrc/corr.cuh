// Persistent correlation kernel: the row pass and the column pass of every
// (window, template pair) unit of one or more in-plane angles in a single launch.
//
// Work items, claimed in increasing order from one atomic counter (lag <= Nu):
//   the row tiles of units 0 .. lag - 1, then for every later unit s
//   [T row tiles of unit s] [T column tiles of unit s - lag], then the column
//   tiles of the last lag units
// with T = l / V tiles of V vectors (V = 16 or 8, CorrCfg).  A row tile takes V
// spectrum rows of unit u: S = W_w conj(P_p), inverse FFT along x (the
// four-step l = 16 N2 transform of fastfft.cuh), written to scratch map slot
// u % S (for odd N2 prime-factor transforms along both axes, CorrCfg::kPfa).
// A column tile takes V columns of that map: inverse FFT along y and the score
// epilogue (border-masked peak and its position, sum of squares, for both
// templates of the pair), reduced into the unit's accumulators; the last
// column tile of a unit computes the two scores, taking the maps' plain sums
// from the spectrum's DC term (sum of the map = L^2 S(0, 0)).
//
// Dependencies and why they cannot deadlock: a column tile of u waits until
// all T row tiles of u are done; a row tile of u >= S waits until all
// column tiles of u - S are done (its scratch slot is free).  Completion is
// counted per tile: after the CTA barrier that ends a tile, one thread (the
// publisher, the CTA's last thread, which has the lightest share of step 1
// when the tasks do not divide evenly) increments the unit's counter, so a
// pass of a unit is done at T increments, claims the CTA's next-but-one item
// (written into the CTA's ring of claimed items just before the following
// barrier, so its warp does not wait for the atomic), and each warp checks the
// dependency of its CTA's next item itself before starting it.  (Counting
// every warp's share before the barrier instead costs each warp a release:
// window 256 8.99 against 8.54 ms, 512 8.54 against 8.18, 768 22.2 against
// 20.6, 20 to 35 k units.)  Both dependencies point at
// items that come earlier in the claim order, and an item is claimed only by
// a running CTA that finishes and publishes it before it waits for anything
// later, so the earliest unpublished item can always proceed.  Every wait is
// bounded; a wait that gives up raises the error flag (reported as
// GS_ERR_TIMEOUT) and the item still completes and is published, so no other
// CTA is left waiting on it.  The units whose maps the wait was for score NaN: it
// adds NaN to their sums (gs_correlate_window_noalloc does not wait for its launches
// and has no other way to tell).  That part of a wait is a call of its own: within
// the loop it cost 1.5 % at windows 128 and 512, and looking at the flag where a
// unit is scored 0.4 % at 720.
//
// Memory ordering: producers store the maps bypassing L1 (st.global with an
// L2 cache hint) and add their accumulator atomics; the CTA barrier that ends
// the tile orders every thread's stores before the
// release increment (acquire-release for column tiles, whose last increment also
// computes the unit's scores), which therefore makes all of them visible
// (release is cumulative).  On the consumer side lane 0 of each warp spins with
// ld.acquire.gpu and __syncwarp() extends the acquire to its warp, whose
// threads read the maps with L1::no_allocate loads (L2, never a stale L1
// line from an earlier occupant of the slot).  A column tile costs two CTA
// barriers (step 1 -> step 2 of the FFT, whose vectors are columns spread
// over all warps for coalesced loads, and the end-of-item barrier); a row
// tile only the end-of-item barrier, as each warp owns two whole rows.
#pragma once

#include <algorithm>
#include <vector>

#include "fastfft.cuh"

namespace gs {

struct CorrArgs {
    const float2* W;         // window spectra, Nw x L2
    const float2* P;         // template-pair spectra of the launch's angles, (angles x pairs) x L2
    float2* R;               // scratch ring, S x L2
    const float2* tw;        // exp(-2 pi i k / l), k < l (even N2 only)
    const int2* unit_wp;     // unit -> (window, angle x pairs + pair)
    int* done_rows;          // per unit, row tiles finished
    int* done_cols;          // per unit, column tiles finished
    UnitAcc* acc;            // per unit, 2 templates
    UnitOut* out;            // results, index angle * out_stride + w * ntmpl + J
    int* next_item;          // claim counter
    int* error;              // set when a bounded wait gives up
    int nu, ntmpl, S, lag;
    long long L2;
    int yb0, yb1;            // border interval of unshifted indices (both axes)
    int pairs;               // template pairs per angle
    long long out_stride;    // results per angle (windows x templates)
    // norm_type 1 (kCorrMoments, kCorrBlocks) instead of acc and out:
    float2* moments;           // per window and map pixel: sums, then (mean, 1 / deviation)
    unsigned long long* keys;  // per angle, window, template: nblk block maxima
    int nblk, nw;
    float inv_l2;
};

// Border interval of unshifted indices: X = (x + l/2) mod l is masked when X <
// d_m/4 or X > l - d_m/4 (GPU_func.cu:681).  Bounds outside the window are brought
// to its edge before they become integers, so that any positive d_m masks what
// it says, one that rounds away and infinity too.
inline void corr_border(CorrArgs* a, float d_m, int l) {
    const float q_lo = d_m / 4.0f, q_hi = (float)l - q_lo;
    const int h = l / 2;
    a->yb0 = (int)floorf(fminf(fmaxf(q_hi, -1.0f), (float)(l - 1))) - h + 1;
    a->yb1 = (int)ceilf(fminf(q_lo, (float)l)) + h - 1;
    if (a->yb1 < a->yb0) a->yb0 = a->yb1 = -1;  // no index
}

// Lag of the column tiles in units for `ctas` resident CTAs and units of `tiles`
// tiles a pass: 2.5 times as many items as CTAs.
inline int corr_lag(int ctas, int tiles) { return (5 * ctas + 4 * tiles - 1) / (4 * tiles); }

// Slots and lags that the autotuner tries around a window's own ring: fixed ones
// where the ring is (`fixed`: windows 512, 720 and 768), else in proportion, since
// rings that go by the resident CTAs have up to some hundred slots.
struct CorrRingTrials {
    std::vector<int> slots, lags;
};
inline CorrRingTrials corr_ring_trials(int slots, int lag, bool fixed) {
    CorrRingTrials t;
    if (fixed) {
        t.slots = {8, 12, 16, 24, 32};
        t.lags = {2, 4, 6, 10};
        return t;
    }
    for (int f : {5, 7, 14, 20}) {
        t.slots.push_back(std::max(2, slots * f / 10));
        t.lags.push_back(std::max(1, lag * f / 10));
    }
    return t;
}
inline int corr_ring_most(int slots, bool fixed) { return fixed ? std::max(32, slots) : 2 * slots; }

// What the column tiles do with the maps: score them; add them into the
// per-pixel moments; z-score them and keep every 1024-element block's maximum.
enum CorrEpi { kCorrScore, kCorrMoments, kCorrBlocks };

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The calling thread waits until *p >= target (bounded: about a second or
// more, then it flags the error and gives up: false).  A barrier must follow before
// other threads rely on the condition.  (Its caller has looked; looking once more
// before sleeping is worth 1.3 % at window 720.)
__device__ __forceinline__ bool wait_counter(const int* p, int target, int* error) {
    if (ld_acquire_gpu(p) >= target) return true;
    bool ok = false;
    for (int it = 0; it < (1 << 22) && !ok; ++it) {
        __nanosleep(256);
        ok = ld_acquire_gpu(p) >= target;
    }
    if (!ok) atomicExch(error, 1);
    return ok;
}

// b^-1 mod m for gcd(b, m) = 1 (compile time, m small)
constexpr int inv_mod(int b, int m) {
    for (int x = 1; x < m; ++x)
        if ((b * x) % m == 1) return x;
    return m == 1 ? 0 : -1;
}

// Tile geometry: V vectors per tile (16 or 8), 16 V threads per CTA (step 2
// has one (vector, k1) task per thread), kThreadsPerSm / (16 V) CTAs per SM (more
// where registers allow).  A pass of one unit is T = L / V tiles.
template <int N2, int V_>
struct CorrCfg {
    static constexpr int L = 16 * N2;
    static constexpr int V = V_;
    static constexpr int BP = (N2 % 2) ? N2 : N2 + 1;  // odd block pitch
    // vector pitch, so that the column tile's stores (V vectors by 16 / V
    // values of n2 in a half-warp) fall into 16 different bank pairs
    static constexpr int VP = 16 * BP + 16 / V;
    static constexpr int kThreads = 16 * V;
    static constexpr int kWarps = kThreads / 32;
    static constexpr int T = L / V;
    // Threads per SM (64, 80 or 128 registers each).  More of them hide more L2
    // latency until the registers no longer hold a task's loads in flight:
    // window 384 (N2 = 24) 241 Gpoint/s with 768 against 208 with 512 and 202
    // with 896; 304 (19) 225 with 1024 against 218 with 768; 320 (20) 221 with
    // 768 against 206 with 1024; 448 (28) 218 with 512 against 195 with 768.
    static constexpr int kThreadsPerSm = N2 <= 19 ? 1024 : N2 <= 26 ? 768 : 512;
    static constexpr int kCtasPerSm = kThreadsPerSm / kThreads;
    static_assert(V == 8 || V == 16, "tile width");
    static_assert(V == 2 * kWarps, "a row tile gives each warp two rows");
    // Odd N2 (l = 720 = 16 x 45): 16 and N2 are coprime, so both passes use
    // the Good-Thomas mapping and need no twiddles between their two DFT
    // steps.  Along x the spectra arrive in that mapping's input order
    // (PfaCols: physical column n2 + N2 n1 holds frequency (N2 n1 + 16 n2)
    // mod L).  Along y the column pass's input row n2 + N2 n1 must hold
    // spectrum row (N2 n1 + 16 n2) mod L, so the row pass reads the spectrum
    // rows in that order.  Either pass's output k1 + 16 k2 is map coordinate
    // (A1 k1 + A2 k2) mod L, A1 = 1 mod 16, 0 mod N2 and A2 = 0 mod 16, 1 mod N2.
    static constexpr bool kPfa = (N2 % 2) == 1;
    static constexpr int A1 = kPfa ? (N2 * inv_mod(N2 % 16, 16)) % L : 1;
    static constexpr int A2 = kPfa ? (16 * inv_mod(16 % N2, N2)) % L : 16;
    // spectrum row that physical row r of the scratch map holds
    __host__ __device__ __forceinline__ static int spectrum_row(int r) {
        if constexpr (kPfa) {
            const int n1 = r / N2, n2 = r - n1 * N2;
            const int q = N2 * n1 + 16 * n2;
            return q < L ? q : q - L;  // N2 n1 + 16 n2 < 2 L
        } else {
            return r;
        }
    }
    // map coordinate of pass output (k1, k2): x of physical column k1 + 16 k2,
    // y of column-pass output k2 of thread k1
    __host__ __device__ static constexpr int map_coord(int k1, int k2) { return (A1 * k1 + A2 * k2) % L; }
};

template <int N2, int V>
struct CorrSmem {
    using C = CorrCfg<N2, V>;
    static constexpr size_t tile = (size_t)C::V * C::VP * sizeof(float2);
    static constexpr size_t tw = C::kPfa ? 0 : (size_t)16 * N2 * sizeof(float2);  // no twiddles with kPfa
    static constexpr size_t bytes = tile + tw + 32;  // and the ring of claimed items
};

// L2 eviction-priority hints: scratch maps are stored "evict last" (they are
// read again shortly) and loaded "evict first" by their only reader; the
// window spectra, reused by every pair of a window block, are loaded
// "evict last".
__device__ __forceinline__ unsigned long long l2_policy_evict_last() {
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ unsigned long long l2_policy_evict_first() {
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float2 ld_l2hint(const float2* ptr, unsigned long long pol) {
    float2 v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;"
                 : "=f"(v.x), "=f"(v.y) : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_l2hint(float2* ptr, float2 v, unsigned long long pol) {
    asm volatile("st.global.L1::no_allocate.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;"
                 :: "l"(ptr), "f"(v.x), "f"(v.y), "l"(pol) : "memory");
}

// Drops one 128-byte line from L2 without writing it back (its contents
// become undefined).  Used on scratch-map lines that have been consumed and
// will be rewritten before they are read again.
__device__ __forceinline__ void l2_discard128(const void* p) {
    asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
}

template <int N2, int V>
__device__ __forceinline__ void corr_row_tile(const CorrArgs& a, int u, int t, float2* tile, const float2* twt,
                                              int2 wp) {
    using F = CorrCfg<N2, V>;
    constexpr int L = F::L;
    const float2* Wr = a.W + (long long)wp.x * a.L2;
    const float2* Pr = a.P + (long long)wp.y * a.L2;
    float2* Rs = a.R + (long long)(u % a.S) * a.L2;
    const int r0 = t * F::V;
    const unsigned long long keep = l2_policy_evict_last();
    // each warp transforms its own two rows (vectors 2w, 2w + 1) through its
    // own part of the tile buffer, so step 1 -> step 2 needs only __syncwarp
    const int w2 = 2 * (threadIdx.x >> 5), lane = threadIdx.x & 31;
    for (int task = lane; task < 2 * N2; task += 32) {
        const int v = w2 + (task >= N2), n2 = task - (task >= N2) * N2;
        const long long base = (long long)F::spectrum_row(r0 + v) * L + n2;
        float2 x[16];
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1)
            x[n1] = cmulc(ld_l2hint(Wr + base + N2 * n1, keep), __ldg(Pr + base + N2 * n1));
        rf::rfft<16, 1, true>(x);
        float2* dst = tile + v * F::VP + n2;
        const float2* tw = twt + n2;
        rf::static_for<16>([&](auto kc) {
            constexpr int k1 = decltype(kc)::value;
            constexpr int r = rf::rpos<16>(k1);
            dst[k1 * F::BP] = (k1 && !F::kPfa) ? cmul(x[r], tw[k1 * N2]) : x[r];
        });
    }
    __syncwarp();
    {
        const int v = threadIdx.x >> 4, k1 = threadIdx.x & 15;  // v = w2 + lane / 16
        float2 b[N2];
        const float2* src = tile + v * F::VP + k1 * F::BP;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) b[n2] = src[n2];
        rf::rfft<N2, 1, true>(b);
        float2* dst = Rs + (long long)(r0 + v) * L + k1;
        rf::static_for<N2>([&](auto kc) {
            constexpr int k2 = decltype(kc)::value;
            st_l2hint(dst + 16 * k2, b[rf::rpos<N2>(k2)], keep);
        });
    }
}

// Border mask of the map rows one column-pass thread produces: bit k2 is set
// when map row map_coord(k1, k2) lies outside the border interval [yb0, yb1]
// (the thread's k1 is fixed for the life of the kernel).
template <int N2, int V>
__device__ __forceinline__ uint2 corr_row_mask(int yb0, int yb1) {
    using F = CorrCfg<N2, V>;
    const int k1 = V == 16 ? (threadIdx.x >> 4) : (threadIdx.x & 15);
    uint2 m = make_uint2(0u, 0u);
    for (int k2 = 0; k2 < N2; ++k2) {
        const int y = F::map_coord(k1, k2);
        if ((unsigned)(y - yb0) > (unsigned)(yb1 - yb0)) {
            if (k2 < 32) m.x |= 1u << k2;
            else m.y |= 1u << (k2 - 32);
        }
    }
    return m;
}

// norm_type 1, sweep 1: cc / l^2 and its square of both templates added into
// the window's per-pixel sums (add_CCG_to_sum, GPU_func.cu:617-633), one 8-byte
// reduction per pixel.  b: the thread's map column x, rows map_coord(k1, k2).
template <int N2, int V>
__device__ __forceinline__ void corr_moments(const CorrArgs& a, int u, int x, int k1, const float2 (&b)[N2]) {
    using F = CorrCfg<N2, V>;
    constexpr int L = F::L, h = L / 2;
    const int2 wp = __ldg(a.unit_wp + u);
    const bool two = 2 * (wp.y % a.pairs) + 1 < a.ntmpl;
    const float s = ((L / 2) % 2 == 0) ? a.inv_l2 : -a.inv_l2;
    float2* mom = a.moments + (long long)wp.x * a.L2 + (x + h < L ? x + h : x - h);
    rf::static_for<N2>([&](auto kc) {
        constexpr int k2 = decltype(kc)::value;
        const float2 c = cscale(b[rf::rpos<N2>(k2)], s);
        const int y = F::map_coord(k1, k2), Y = y + h < L ? y + h : y - h;
        atomicAdd(mom + (long long)Y * L, two ? make_float2(c.x + c.y, fmaf(c.y, c.y, c.x * c.x)) : make_float2(c.x, c.x * c.x));
    });
}

// norm_type 1, sweep 2: z-scores against the window's per-pixel (mean, 1 /
// deviation), 0 where that is marked negative (no positive deviation), and the
// maximum of every 1024-element block of the flat map (update_CCG +
// get_peak_pos, GPU_func.cu:648-662, 711-745).  The product rounds as the
// reference's division does: 1 / deviation is rounded once, from double, where the
// deviation was (dividing instead took norm_type 1 at window 512 from 6.2 to
// 8.0 ms); the rounding of 1 / l^2 is in the maps of both sweeps and cancels.
// The tile's z go through the tile buffer as float_order keys (l rows of 16, both
// templates), so that a thread takes a whole 16-column run of one row, which lies
// inside one block (l is a multiple of 32); runs of one block in neighbouring lanes
// are combined before the one atomic.  One atomic per map value instead cost 173
// us per 12 pairs at window 512.  The 16-byte pieces of a row are rotated by its
// index to keep both sides free of bank conflicts.
template <int N2, int V>
__device__ __forceinline__ void corr_blocks(const CorrArgs& a, int u, int v, int x, int k1, const float2 (&b)[N2],
                                            unsigned* z) {
    using F = CorrCfg<N2, V>;
    static_assert(V == 16 && !F::kPfa, "16-column runs in natural order");
    constexpr int L = F::L, h = L / 2;
    const int2 wp = __ldg(a.unit_wp + u);
    const int an = wp.y / a.pairs, p = wp.y - an * a.pairs;
    const float s = ((L / 2) % 2 == 0) ? a.inv_l2 : -a.inv_l2;
    const int X = x + h < L ? x + h : x - h;
    const float2* mom = a.moments + (long long)wp.x * a.L2 + X;
    __syncthreads();  // every read of the tile's columns is done
    rf::static_for<N2>([&](auto kc) {
        constexpr int k2 = decltype(kc)::value;
        const int y = k1 + 16 * k2, Y = y + h < L ? y + h : y - h;
        const float2 m = __ldg(mom + (long long)Y * L);
        const float2 c = cscale(b[rf::rpos<N2>(k2)], s);
        unsigned* o = z + Y * 16 + (((v >> 2) ^ ((Y >> 1) & 3)) << 2) + (v & 3);
        o[0] = float_order(m.y >= 0.0f ? (c.x - m.x) * m.y : 0.0f);
        o[L * 16] = float_order(m.y >= 0.0f ? (c.y - m.x) * m.y : 0.0f);
    });
    __syncthreads();
    const int X0 = X & ~15;  // V = 16: the tile's columns start at a multiple of 16
    for (int r = threadIdx.x; r < 2 * L; r += F::kThreads) {  // L is a multiple of 32: no partial warps
        const int q = r >= L, Y = q ? r - L : r, J = 2 * p + q;
        const uint4* row = reinterpret_cast<const uint4*>(z + (q * L + Y) * 16);
        unsigned best = 0u;
        int at = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 w = row[c ^ ((Y >> 1) & 3)];
            if (w.x > best) { best = w.x; at = 4 * c; }
            if (w.y > best) { best = w.y; at = 4 * c + 1; }
            if (w.z > best) { best = w.z; at = 4 * c + 2; }
            if (w.w > best) { best = w.w; at = 4 * c + 3; }
        }
        const int pos = Y * L + X0 + at, blk = (Y * L + X0) >> 10;
        unsigned long long key = ((unsigned long long)best << 32) | (unsigned)~pos;
        // rows of one block sit in neighbouring lanes (a warp holds rows of one template)
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            if (o * L >= 1024) break;
            const unsigned long long k = __shfl_down_sync(0xffffffffu, key, o);
            const int kb = __shfl_down_sync(0xffffffffu, blk, o);
            if ((threadIdx.x & 31) + o < 32 && kb == blk) key = k > key ? k : key;
        }
        const int before = __shfl_up_sync(0xffffffffu, blk, 1);
        if (J < a.ntmpl && ((threadIdx.x & 31) == 0 || before != blk))
            atomicMax(a.keys + (((long long)an * a.nw + wp.x) * a.ntmpl + J) * a.nblk + blk, key);
    }
}

template <int N2, int V, CorrEpi kEpi>
__device__ __forceinline__ void corr_col_tile(const CorrArgs& a, int u, int t, float2* tile, const float2* twt,
                                              uint2 ymask) {
    using F = CorrCfg<N2, V>;
    constexpr int L = F::L;
    constexpr int h = L / 2;
    const float2* Rs = a.R + (long long)(u % a.S) * a.L2;
    const int c0 = t * F::V;
    const unsigned long long drop = l2_policy_evict_first();
    for (int task = threadIdx.x; task < F::V * N2; task += F::kThreads) {
        const int n2 = task / F::V, v = task - n2 * F::V;
        const float2* src = Rs + (long long)n2 * L + c0 + v;
        float2 x[16];
#pragma unroll
        for (int n1 = 0; n1 < 16; ++n1) x[n1] = ld_l2hint(src + (long long)N2 * n1 * L, drop);
        rf::rfft<16, 1, true>(x);
        float2* dst = tile + v * F::VP + n2;
        const float2* tw = twt + n2;
        rf::static_for<16>([&](auto kc) {
            constexpr int k1 = decltype(kc)::value;
            constexpr int r = rf::rpos<16>(k1);
            dst[k1 * F::BP] = (k1 && !F::kPfa) ? cmul(x[r], tw[k1 * N2]) : x[r];
        });
    }
    __syncthreads();
    // every line of this tile's 16 columns has been read (the barrier orders
    // the loads before the discards): drop them from L2 instead of letting
    // them be written back; the slot is rewritten before its next read.  An
    // 8-column tile owns only half of each line and leaves them alone.
    if (V == 16)
        for (int r = threadIdx.x; r < L; r += F::kThreads) l2_discard128(Rs + (long long)r * L + c0);
    // step-2 task: (vector, k1); both orders read distinct banks per half-warp
    // for their width
    const int v = V == 16 ? (threadIdx.x & 15) : (threadIdx.x >> 4);
    const int k1 = V == 16 ? (threadIdx.x >> 4) : (threadIdx.x & 15);
    // map column held by physical column c0 + v (the row pass's output order)
    const int x = F::kPfa ? F::map_coord((c0 + v) & 15, (c0 + v) >> 4) : c0 + v;
    // column outside the border: the rows of ymask count, else none
    if ((unsigned)(x - a.yb0) <= (unsigned)(a.yb1 - a.yb0)) ymask = make_uint2(0u, 0u);
    if constexpr (kEpi != kCorrScore) {
        float2 b[N2];
        const float2* src = tile + v * F::VP + k1 * F::BP;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) b[n2] = src[n2];
        rf::rfft<N2, 1, true>(b);
        if constexpr (kEpi == kCorrMoments) corr_moments<N2, V>(a, u, x, k1, b);
        else corr_blocks<N2, V>(a, u, v, x, k1, b, reinterpret_cast<unsigned*>(tile));
        return;
    }
    constexpr float sgn = ((L / 2) % 2 == 0) ? 1.0f : -1.0f;
    // Per point the border-masked maximum with its k2 and the sum of squares;
    // the map's plain sum is L^2 times its spectrum's DC term, taken when the
    // unit's scores are computed.
    float best1 = 0.0f, best2 = 0.0f;   // reference peak = max(0, masked max)
    int bk1 = -1, bk2 = -1;
    float2 s2 = make_float2(0.0f, 0.0f);
    {
        float2 b[N2];
        const float2* src = tile + v * F::VP + k1 * F::BP;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) b[n2] = src[n2];
        rf::rfft<N2, 1, true>(b);
        rf::static_for<N2>([&](auto kc) {
            constexpr int k2 = decltype(kc)::value;
            const float2 val = b[rf::rpos<N2>(k2)];
            const bool in = (((k2 < 32 ? ymask.x : ymask.y) >> (k2 & 31)) & 1u) != 0u;
            const float v1 = sgn * val.x, v2 = sgn * val.y;
            const bool g1 = in && v1 > best1, g2 = in && v2 > best2;
            best1 = g1 ? v1 : best1;
            bk1 = g1 ? k2 : bk1;
            best2 = g2 ? v2 : best2;
            bk2 = g2 ? k2 : bk2;
            s2 = __ffma2_rn(val, val, s2);
        });
    }
    // Warp reductions: the peaks by integer reductions of the value bits (the
    // peaks are not negative) and then of the smallest map index that has
    // the value (within one thread, the first in k2 order); the sums in double,
    // each half of the warp taking one template's after one exchange.  Shuffles
    // share the pipe of the shared-memory exchange, the tighter one here.
    const int X = x + h < L ? x + h : x - h;
    auto map_index = [&](int k2) {
        const int y = F::map_coord(k1, k2);
        return (unsigned)((y + h < L ? y + h : y - h) * L + X);
    };
    const unsigned m1 = __float_as_uint(best1), m2 = __float_as_uint(best2);
    const unsigned p1 = __reduce_max_sync(0xffffffffu, m1), p2 = __reduce_max_sync(0xffffffffu, m2);
    const unsigned i1 = __reduce_min_sync(0xffffffffu, bk1 >= 0 && m1 == p1 ? map_index(bk1) : 0xffffffffu);
    const unsigned i2 = __reduce_min_sync(0xffffffffu, bk2 >= 0 && m2 == p2 ? map_index(bk2) : 0xffffffffu);
    const int lane = threadIdx.x & 31;
    const bool second = lane >= 16;
    double d = (second ? (double)s2.y : (double)s2.x) + __shfl_xor_sync(0xffffffffu, second ? (double)s2.x : (double)s2.y, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    // one set of atomics per warp (published with the tile)
    if ((lane & 15) == 0) {
        UnitAcc* ac = a.acc + 2 * (long long)u + (second ? 1 : 0);
        const unsigned peak = second ? p2 : p1;
        if (peak) atomicMax(&ac->key, ((unsigned long long)peak << 32) | (unsigned long long)(~(second ? i2 : i1)));
        atomicAdd(&ac->s2, d);
    }
}

// Score of one template from its accumulators (main.cu:869-876); s1 is the
// sum of the whole map.
__device__ __forceinline__ UnitOut unit_score(const UnitAcc& ac, double s1, int l) {
    const float peak = key_value(ac.key);
    UnitOut u;
    u.peak = peak;
    u.pos = key_index(ac.key);
    const double ra = s1 - peak;
    const double rb = ac.s2 - (double)peak * peak;
    const double rc = (double)l * l - 1.0;
    const double sd = sqrt(rb / rc - (ra / rc) * (ra / rc));
    u.sigma = (float)sd;
    u.score = sd > 0.0 ? (float)(peak / sd) : __int_as_float(0x7fc00000);
    return u;
}
__device__ __forceinline__ UnitOut unit_score(const UnitAcc& ac, int l) { return unit_score(ac, ac.s1, l); }

// Item indices of one persistent launch over n units (2 x l/8 tiles per unit)
// must fit an int.
inline bool corr_units_fit(int l, long long n) { return n < (1ll << 31) && (n + 64) * 2 * (l / 8) < (1ll << 31); }

// Whether a claim is one of the launch's `total` items.  Every CTA claims two items
// past the last one, more in all than the room that corr_units_fit leaves
// below 2^31 at windows under 160: such a claim is negative, and no item either.
__host__ __device__ __forceinline__ bool corr_claimed(int item, int total) { return (unsigned)item < (unsigned)total; }

// What a claimed item is.
struct CorrItem {
    int u, j;  // unit, tile
    bool row;
};

template <int T>
__host__ __device__ __forceinline__ CorrItem corr_item(const CorrArgs& a, int item) {
    const int head = a.lag * T;
    if (item < head) return CorrItem{item / T, item % T, true};
    const int i = item - head, s = i / (2 * T), j = i - s * (2 * T);
    if (s < a.nu - a.lag) return j < T ? CorrItem{a.lag + s, j, true} : CorrItem{s, j - T, false};
    const int c = i - (a.nu - a.lag) * (2 * T);
    return CorrItem{a.nu - a.lag + c / T, c % T, false};
}

// The rest of a wait whose counter was not there at once.  Where it gives up, units u
// and v (v < 0: none) are scored NaN.
static __device__ __noinline__ void corr_wait_slow(const int* p, int target, int* error, UnitAcc* acc, int u, int v) {
    if (wait_counter(p, target, error) || !acc) return;
    for (int q = 0; q < 2; ++q) {
        atomicAdd(&acc[2 * (long long)u + q].s2, __longlong_as_double(0x7ff8000000000000ll));
        if (v >= 0) atomicAdd(&acc[2 * (long long)v + q].s2, __longlong_as_double(0x7ff8000000000000ll));
    }
    __threadfence();  // before anything the item overwrites too early
}

// Each warp waits for what an item depends on before working on it (lane 0 looks,
// __syncwarp() extends its acquire to the warp): a row tile for its slot's previous
// unit's column tiles, a column tile for its unit's row tiles.
template <int T, CorrEpi kEpi>
__device__ __forceinline__ void corr_wait_for(const CorrArgs& a, const CorrItem& it) {
    UnitAcc* acc = kEpi == kCorrScore ? a.acc : nullptr;
    if (!it.row) {
        if ((threadIdx.x & 31) == 0 && ld_acquire_gpu(a.done_rows + it.u) < T)
            corr_wait_slow(a.done_rows + it.u, T, a.error, acc, it.u, -1);
        __syncwarp();
    } else if (it.u >= a.S) {
        if ((threadIdx.x & 31) == 0 && ld_acquire_gpu(a.done_cols + (it.u - a.S)) < T)
            corr_wait_slow(a.done_cols + (it.u - a.S), T, a.error, acc, it.u, it.u - a.S);
        __syncwarp();
    }
}

// Count a finished tile; the last count of a unit's column pass computes its
// two scores.
template <int N2, int V, CorrEpi kEpi>
__device__ __forceinline__ void corr_publish(const CorrArgs& a, const CorrItem& it) {
    using F = CorrCfg<N2, V>;
    const int u = it.u;
    if (it.row) {
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&a.done_rows[u]) : "memory");
        return;
    }
    if constexpr (kEpi != kCorrScore) {
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&a.done_cols[u]) : "memory");
        return;
    }
    int prev;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(prev) : "l"(&a.done_cols[u]) : "memory");
    if (prev != F::T - 1) return;
    const int2 wp = a.unit_wp[u];
    const UnitAcc* ac = a.acc + 2 * (long long)u;
    // sum of the map c1 + i c2 = L^2 S(0, 0), S = W conj(P)
    // (frequency (0, 0) sits at element 0 in either column order)
    const float2 w0 = __ldg(a.W + (long long)wp.x * a.L2);
    const float2 p0 = __ldg(a.P + (long long)wp.y * a.L2);
    const double sg = ((F::L / 2) % 2 == 0) ? 1.0 : -1.0;
    const double l2 = (double)a.L2;
    const double sums[2] = {sg * l2 * ((double)w0.x * p0.x + (double)w0.y * p0.y),
                            sg * l2 * ((double)w0.y * p0.x - (double)w0.x * p0.y)};
    for (int q = 0; q < 2; ++q) {
        const long long o = unit_out_index(wp.y, q, wp.x, a.pairs, a.ntmpl, a.out_stride);
        if (o < 0) break;
        UnitAcc v;
        v.key = __ldcg(&ac[q].key);
        v.s2 = __ldcg(&ac[q].s2);
        a.out[o] = unit_score(v, sums[q], F::L);
    }
}

template <int N2, int V, CorrEpi kEpi = kCorrScore>
__global__ void __launch_bounds__(CorrCfg<N2, V>::kThreads, CorrCfg<N2, V>::kCtasPerSm) k_corr_persistent(CorrArgs a) {
    using F = CorrCfg<N2, V>;
    using SM = CorrSmem<N2, V>;
    constexpr int kPub = F::kThreads - 1;  // the publisher
    extern __shared__ __align__(16) unsigned char smc[];
    float2* tile = reinterpret_cast<float2*>(smc);
    float2* twt = reinterpret_cast<float2*>(smc + SM::tile);
    int* ish = reinterpret_cast<int*>(smc + SM::tile + SM::tw);  // ring of 4 claimed items
    // inverse twiddles W_L^{-n2 k1} = exp(+2 pi i n2 k1 / L), table [k1][n2]
    for (int i = threadIdx.x; i < (F::kPfa ? 0 : 16 * N2); i += F::kThreads) {
        const int k1 = i / N2, n2 = i - k1 * N2;
        twt[i] = twiddle(a.tw, n2 * k1, true);
    }
    const uint2 ymask = corr_row_mask<N2, V>(a.yb0, a.yb1);
    const int total = a.nu * 2 * F::T;
    // the CTA always holds its current item and the next one
    if (threadIdx.x == kPub) {
        ish[0] = atomicAdd(a.next_item, 1);
        ish[1] = atomicAdd(a.next_item, 1);
    }
    __syncthreads();
    int item = ish[0];
    int claimed = 0;  // the publisher's claim for slot (iter + 1) & 3, made after the previous barrier
    for (int iter = 0; corr_claimed(item, total); ++iter) {
        // the unit's (window, pair) is read-only in this launch: its load is
        // issued before the dependency wait and overlaps it
        const CorrItem it = corr_item<F::T>(a, item);
        const int2 wp = it.row ? __ldg(a.unit_wp + it.u) : make_int2(0, 0);
        corr_wait_for<F::T, kEpi>(a, it);
        if (it.row) corr_row_tile<N2, V>(a, it.u, it.j, tile, twt, wp);
        else corr_col_tile<N2, V, kEpi>(a, it.u, it.j, tile, twt, ymask);
        // the claim made after the previous barrier enters the ring only now,
        // so the publisher's warp did not wait for the atomic's return
        if (threadIdx.x == kPub && iter > 0) ish[(iter + 1) & 3] = claimed;
        // every thread is done with the item: the tile buffer is free, the
        // item's stores and atomics are ordered before its publication, and
        // slot (iter + 1) & 3 holds the next item; slot (iter + 2) & 3 was
        // last read two iterations ago
        __syncthreads();
        const int next = ish[(iter + 1) & 3];
        if (threadIdx.x == kPub) {
            corr_publish<N2, V, kEpi>(a, it);
            claimed = atomicAdd(a.next_item, 1);  // for slot (iter + 2) & 3
        }
        item = next;
    }
}

}  // namespace gs
