// Float32 running sums in their exact sequential order, computed in parallel.
//
// The search's hot-pixel bounds come from two float32 sums over the micrograph
// taken pixel by pixel (main.cu:530-535); float addition is not associative,
// so the order is part of the result.  One dependent addition per pixel costs
// 4 cycles of latency: 73.4 ms for 5760 x 4092 pixels when a single thread does
// it, with the rest of the GPU waiting; this way it is 6.7 ms.
//
// While the running sum s stays inside one binade [2^e, 2^(e+1)) it is k u with
// u = 2^(e-23) and an integer k, and rounding to nearest even makes adding q
//     k <- k + rint(q / u)
// where k matters only when q / u is exactly halfway between two integers: the
// neighbour that makes the new k even is taken.  So a run of terms is a map
// k -> k + d (k even) or k + d + o (k odd), o in {-1, 0, 1}, and such maps
// compose associatively: they can be computed for short runs in parallel,
// combined in a tree, and applied at once as long as the smallest and largest
// k on the way stay inside the binade.  Runs where they might not are added
// term by term.
#pragma once

#include "common.cuh"

namespace gs {

// A run of terms in units of the binade's last place.
struct SeqRun {
    int d;       // change of k from an even k
    int o;       // extra change from an odd k
    int mn, mx;  // bounds of the change on the way, up to 1 (see seq_apply)
};
constexpr int kSeqFail = 1 << 28;  // mx of a run that cannot be applied as a whole
constexpr int kSeqRange = 1 << 24;

__host__ __device__ __forceinline__ SeqRun seq_identity() { return SeqRun{0, 0, 0, 0}; }

__host__ __device__ __forceinline__ unsigned seq_bits(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v);
#else
    unsigned u;
    memcpy(&u, &v, 4);
    return u;
#endif
}
__host__ __device__ __forceinline__ float seq_float(unsigned u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float v;
    memcpy(&v, &u, 4);
    return v;
#endif
}

// Sign and exponent of s, or 0 when runs cannot be applied to it (zero, tiny,
// huge, infinite or NaN).
__host__ __device__ __forceinline__ unsigned seq_binade(float s) {
    const unsigned b = seq_bits(s) >> 23, e = b & 0xffu;
    return e >= 30u && e <= 250u ? b : 0u;
}

// 1 / u with the sign of the sum: q times it is q in units of the last place,
// positive towards larger |s|.  An exact power of two for exponents 30 to 250.
__host__ __device__ __forceinline__ float seq_scale(unsigned binade) {
    const unsigned e = binade & 0xffu;
    return seq_float(((binade >> 8) << 31) | ((277u - e) << 23));
}

// The run of N terms.  Terms of 2^22 units and more (and NaN) make it fail.
template <int N>
__host__ __device__ __forceinline__ SeqRun seq_run(const float (&q)[N], float scale) {
    constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23: adding it rounds to an integer
    int acc = 0, o = 0, mn = 0, mx = 0;
    float big = 0.0f;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < N; ++i) {
        const float x = q[i] * scale;
#ifdef __CUDA_ARCH__
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(big) : "f"(fabsf(x)));
        const float y = __fadd_rn(x, kMagic);
        const float r = __fsub_rn(y, kMagic);
        const float f = __fsub_rn(x, r);
#else
        if (!(fabsf(x) <= big) && big == big) big = fabsf(x);  // keeps a NaN
        volatile float yv = x + kMagic;
        const float y = yv;
        volatile float rv = y - kMagic;
        const float r = rv, f = x - r;
#endif
        int step = (int)(seq_bits(y) - 0x4b400000u);
        if (fabsf(f) == 0.5f) {
            // halfway: `step` is the even neighbour, the other one makes an odd k even
            const int other = step + (f > 0.0f ? 1 : -1);
            const int se = (acc & 1) ? other : step;
            const int so = ((acc + o) & 1) ? step : other;  // k odd at the start
            o += so - se;
            step = se;
        }
        acc += step;
        mn = acc < mn ? acc : mn;
        mx = acc > mx ? acc : mx;
    }
    if (!(big < 4194304.0f) || mn < -kSeqRange || mx > kSeqRange) return SeqRun{0, 0, 0, kSeqFail};
    return SeqRun{acc, o, mn, mx};
}

// Run a, then run b.
__host__ __device__ __forceinline__ SeqRun seq_then(const SeqRun& a, const SeqRun& b) {
    const int ao = a.d + a.o;
    const int e = a.d + b.d + ((a.d & 1) ? b.o : 0);
    const int f = ao + b.d + ((ao & 1) ? 0 : b.o);
    SeqRun r;
    r.d = e;
    r.o = f - e;
    // b's bounds hold for its even start and up to 1 for its odd one
    r.mn = min(a.mn, a.d + b.mn - 1);
    r.mx = max(a.mx, a.d + b.mx + 1);
    if (a.mx >= kSeqFail || b.mx >= kSeqFail || r.mn < -kSeqRange || r.mx > kSeqRange) r = SeqRun{0, 0, 0, kSeqFail};
    return r;
}

// Applies a run computed for seq_scale(binade) to s; false (s untouched)
// when s has left that binade or might leave it on the way.
__host__ __device__ __forceinline__ bool seq_apply(float& s, unsigned binade, const SeqRun& r) {
    const unsigned b = seq_bits(s);
    if (binade == 0u || b >> 23 != binade || r.mx >= kSeqFail) return false;
    const int k = (int)((b & 0x7fffffu) | 0x800000u);
    if (k + r.mn - 1 <= 0x800000 || k + r.mx + 1 >= 0x1000000) return false;
    const int n = k + r.d + ((k & 1) ? r.o : 0);
    s = seq_float((binade << 23) | ((unsigned)n & 0x7fffffu));
    return true;
}

// sums[b] = ((0 + q_b[0]) + q_b[1]) + ... for the two arrays q_0 = q and
// q_1 = q + stride (16-byte aligned), one CTA each.
//
// Bound by the FP32 and integer issue rate of the one SM each sum runs on
// (about 11 instructions a term).  A block of 16384 terms (16 a thread) is
// staged by cp.async while the one before it is summed; each warp's 512-term
// run, composed by shuffles, is a unit that is either applied or added term
// by term by one thread.  Chunks of 20 floats keep both the 16-byte copies
// aligned and a thread's 16-byte reads free of bank conflicts.
constexpr int kSeqThreads = 1024;
constexpr int kSeqTerms = 16;                         // per thread
constexpr int kSeqPitch = kSeqTerms + 4;
constexpr int kSeqBlock = kSeqThreads * kSeqTerms;
constexpr size_t kSeqSmem = 2 * (size_t)kSeqThreads * kSeqPitch * sizeof(float);

__device__ __forceinline__ void seq_stage(float* buf, const float* __restrict__ q, long long base, long long n) {
#pragma unroll
    for (int j = 0; j < kSeqTerms / 4; ++j) {
        const int i4 = j * kSeqThreads + threadIdx.x;  // 16-byte piece
        const long long g = base + 4ll * i4;
        const long long left = n - g;
        const int bytes = left >= 4 ? 16 : left > 0 ? (int)left * 4 : 0;  // the rest is zero filled: s + 0 = s
        const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + (i4 >> 2) * kSeqPitch + (i4 & 3) * 4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(q + (bytes ? g : 0)), "r"(bytes)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ SeqRun seq_shfl_down(const SeqRun& r, int off) {
    SeqRun v;
    v.d = __shfl_down_sync(0xffffffffu, r.d, off);
    v.o = __shfl_down_sync(0xffffffffu, r.o, off);
    v.mn = __shfl_down_sync(0xffffffffu, r.mn, off);
    v.mx = __shfl_down_sync(0xffffffffu, r.mx, off);
    return v;
}

// Lane 0 gets the composition of all 32 lanes' runs in lane order.
__device__ __forceinline__ SeqRun seq_warp(SeqRun r) {
#pragma unroll
    for (int off = 1; off < 32; off *= 2) r = seq_then(r, seq_shfl_down(r, off));
    return r;
}

__global__ void __launch_bounds__(kSeqThreads) k_seq_sums(const float* __restrict__ q, long long stride, long long n,
                                                          float* __restrict__ sums) {
    extern __shared__ __align__(16) float seq_buf[];
    __shared__ SeqRun runs[32];
    __shared__ float sh_s;
    __shared__ int sh_w;
    q += blockIdx.x * stride;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh_s = 0.0f;
    seq_stage(seq_buf, q, 0, n);
    int cur = 0;
    for (long long base = 0; base < n; base += kSeqBlock, cur ^= 1) {
        const float* buf = seq_buf + cur * kSeqThreads * kSeqPitch;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the block is staged, and the other buffer free
        if (base + kSeqBlock < n) seq_stage(seq_buf + (cur ^ 1) * kSeqThreads * kSeqPitch, q, base + kSeqBlock, n);
        float t[kSeqTerms];
#pragma unroll
        for (int j = 0; j < kSeqTerms / 4; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(buf + threadIdx.x * kSeqPitch + 4 * j);
            t[4 * j] = v.x; t[4 * j + 1] = v.y; t[4 * j + 2] = v.z; t[4 * j + 3] = v.w;
        }
        int w0 = 0;  // warps before it are in the sum
        do {
            const unsigned binade = seq_binade(sh_s);
            SeqRun r = seq_identity();
            if (warp >= w0 && binade) r = seq_warp(seq_run(t, seq_scale(binade)));
            if (lane == 0) runs[warp] = r;
            __syncthreads();
            if (warp == 0) {
                const SeqRun all = seq_warp(runs[lane]);
                if (lane == 0) {
                    float s = sh_s;
                    int w = 32;
                    if (!seq_apply(s, binade, all)) {
                        for (w = w0; w < 32; ++w) {
                            if (seq_apply(s, binade, runs[w])) continue;
                            const float4* v = reinterpret_cast<const float4*>(buf + w * 32 * kSeqPitch);
#pragma unroll 4
                            for (int c = 0; c < 32; ++c)
#pragma unroll
                                for (int j = 0; j < kSeqTerms / 4; ++j) {
                                    const float4 a = v[c * (kSeqPitch / 4) + j];
                                    s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
                                }
                            if (seq_binade(s) != binade) {  // the later warps' runs need another unit
                                ++w;
                                break;
                            }
                        }
                    }
                    sh_s = s;
                    sh_w = w;
                }
            }
            __syncthreads();
            w0 = sh_w;
        } while (w0 < 32);
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = sh_s;
}

}  // namespace gs
