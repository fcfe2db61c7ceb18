// Float32 running sums in their exact sequential order, computed in parallel.
//
// The search's hot-pixel bounds come from two float32 sums over the micrograph
// taken pixel by pixel (main.cu:530-535); float addition is not associative,
// so the order is part of the result.  One dependent addition per pixel costs
// 4 cycles of latency: 73.4 ms for 5760 x 4092 pixels when a single thread does
// it, with the rest of the GPU waiting; this way it is 0.7 ms at a mean of 5 and a
// deviation of 1.2, 1.4 to 2.3 for noise around zero, 18 at a mean of 100 (see
// k_seq_apply).
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

// The run of N terms (N even).  The change of k is summed in floats, exact
// integers below 2^24; on the way k moves by no more than the terms' absolute
// sum and their rounding.  Runs whose absolute sum reaches 2^22 units (or is
// NaN) fail.
template <int N>
__host__ __device__ __forceinline__ SeqRun seq_run(const float (&q)[N], float scale) {
    constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23: adding it rounds to an integer
    float2 acc = make_float2(0.0f, 0.0f);  // of the even and the odd terms
    float size = 0.0f;
    int o = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int i = 0; i < N; i += 2) {
#ifdef __CUDA_ARCH__
        const float2 x = cscale(make_float2(q[i], q[i + 1]), scale);
        const float2 y = cadd(x, make_float2(kMagic, kMagic));
        float2 r = cadd(y, make_float2(-kMagic, -kMagic));
        const float2 f = csub(x, r);
#else
        const float2 x = make_float2(q[i] * scale, q[i + 1] * scale);
        volatile float y0 = x.x + kMagic, y1 = x.y + kMagic;
        float2 r = make_float2(y0 - kMagic, y1 - kMagic);
        const float2 f = make_float2(x.x - r.x, x.y - r.y);
#endif
        size += fabsf(x.x) + fabsf(x.y);
        if (fabsf(f.x) == 0.5f || fabsf(f.y) == 0.5f) {
            // halfway: r is the even neighbour, the other one makes an odd k even
            int k = (int)(acc.x + acc.y);
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int t = 0; t < 2; ++t) {
                const float g = t ? f.y : f.x, v = t ? r.y : r.x;
                const int even = (int)v, other = even + (g > 0.0f ? 1 : -1);
                int step = even;
                if (fabsf(g) == 0.5f) {
                    step = (k & 1) ? other : even;
                    o += (((k + o) & 1) ? even : other) - step;  // k odd at the start
                }
                k += step;
                if (t) r.y = (float)step;
                else r.x = (float)step;
            }
        }
        acc = cadd(acc, r);
    }
    if (!(size < 4194304.0f)) return SeqRun{0, 0, 0, kSeqFail};
    const int far = (int)(size * 1.0001f) + N;
    return SeqRun{(int)(acc.x + acc.y), o, -far, far};
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

// Three launches over blocks of kSeqBlock terms:
//   the terms' kernel (k_mic_quot) also leaves the blocks' sums in double;
//   k_seq_runs, one CTA per block, predicts the binade at the block's start from
//   those sums and composes the block's run for it (threads 16 terms, then
//   warps, then the CTA), all blocks at once;
//   k_seq_apply, one CTA per sum, applies the blocks' runs in order, about 40
//   cycles each.  A block whose binade was predicted wrongly (float sums drift
//   from the exact ones) or that comes too close to its edges is staged in
//   shared memory and done 512 terms at a time by one warp: by a run where that
//   applies, term by term (4 cycles each) where it does not.
// The last kernel is what is left: its time goes with the number of blocks in
// which the sum passes a power of two, 12 of 1438 for a mean of a few deviations and
// 136 for 5760 x 4092 pixels of coloured noise around 0, and in which the float sum
// has drifted into another binade than the exact one: most of them for a mean of a
// hundred deviations, where all terms of a binade round the same way.
constexpr int kSeqThreads = 1024;
constexpr int kSeqTerms = 16;  // per thread
constexpr int kSeqBlock = kSeqThreads * kSeqTerms;
// chunks of 20 floats: 16-byte copies stay aligned and a lane's 16-byte reads
// free of bank conflicts
constexpr int kSeqPitch = kSeqTerms + 4;
constexpr size_t kSeqSmem = (size_t)kSeqThreads * kSeqPitch * sizeof(float);

struct SeqBlock {
    SeqRun run;
    unsigned binade;  // it was composed for; 0: none
};

__device__ __forceinline__ SeqRun seq_shfl_down(const SeqRun& r, int off) {
    SeqRun v;
    v.d = __shfl_down_sync(0xffffffffu, r.d, off);
    v.o = __shfl_down_sync(0xffffffffu, r.o, off);
    v.mn = __shfl_down_sync(0xffffffffu, r.mn, off);
    v.mx = __shfl_down_sync(0xffffffffu, r.mx, off);
    return v;
}

// The composition of all 32 lanes' runs in lane order, in lane 0 at least.
// Without ties and failed runs a prefix sum and two reductions do.
__device__ __forceinline__ SeqRun seq_warp(SeqRun r) {
    if (!__any_sync(0xffffffffu, r.o != 0 || r.mx >= kSeqFail)) {
        const int lane = threadIdx.x & 31;
        int sum = r.d;
#pragma unroll
        for (int off = 1; off < 32; off *= 2) {
            const int v = __shfl_up_sync(0xffffffffu, sum, off);
            if (lane >= off) sum += v;
        }
        const int before = sum - r.d;
        const int mn = __reduce_min_sync(0xffffffffu, before + r.mn), mx = __reduce_max_sync(0xffffffffu, before + r.mx);
        const int d = __shfl_sync(0xffffffffu, sum, 31);
        return mn < -kSeqRange || mx > kSeqRange ? SeqRun{0, 0, 0, kSeqFail} : SeqRun{d, 0, mn, mx};
    }
#pragma unroll
    for (int off = 1; off < 32; off *= 2) r = seq_then(r, seq_shfl_down(r, off));
    return r;
}

// Blocks of the array q + blockIdx.y stride (16-byte aligned), their exact sums at
// exact + blockIdx.y gridDim.x; results at out + blockIdx.y gridDim.x.
__global__ void __launch_bounds__(kSeqThreads) k_seq_runs(const float* __restrict__ q, long long stride, long long n,
                                                          const double* __restrict__ exact, SeqBlock* __restrict__ out) {
    __shared__ SeqRun runs[32];
    __shared__ double red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x;
    q += blockIdx.y * stride;
    exact += (size_t)blockIdx.y * gridDim.x;
    float t[kSeqTerms];
    const long long base = (long long)b * kSeqBlock + threadIdx.x * kSeqTerms;
#pragma unroll
    for (int j = 0; j < kSeqTerms; j += 4) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // behind the end: s + 0 = s
        if (base + j + 3 < n) {
            v = *reinterpret_cast<const float4*>(q + base + j);
        } else {
            if (base + j < n) v.x = q[base + j];
            if (base + j + 1 < n) v.y = q[base + j + 1];
            if (base + j + 2 < n) v.z = q[base + j + 2];
        }
        t[j] = v.x; t[j + 1] = v.y; t[j + 2] = v.z; t[j + 3] = v.w;
    }
    double before[1] = {0.0};
    for (int i = threadIdx.x; i < b; i += kSeqThreads) before[0] += exact[i];
    block_sum<1>(before, red);
    const unsigned binade = seq_binade((float)before[0]);
    SeqRun r = seq_identity();
    if (binade) r = seq_warp(seq_run(t, seq_scale(binade)));
    if (lane == 0) runs[warp] = r;
    __syncthreads();
    if (warp == 0) {
        r = seq_warp(runs[lane]);
        if (lane == 0) out[(size_t)blockIdx.y * gridDim.x + b] = SeqBlock{r, binade};
    }
}

// One block of terms into buf, zeros behind the end.
__device__ __forceinline__ void seq_stage(float* buf, const float* __restrict__ q, long long base, long long n) {
#pragma unroll
    for (int j = 0; j < kSeqTerms / 4; ++j) {
        const int i4 = j * kSeqThreads + threadIdx.x;  // 16-byte piece
        const long long g = base + 4ll * i4;
        const long long left = n - g;
        const int bytes = left >= 4 ? 16 : left > 0 ? (int)left * 4 : 0;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + (i4 >> 2) * kSeqPitch + (i4 & 3) * 4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(q + (bytes ? g : 0)), "r"(bytes)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// sums[b] = ((0 + q_b[0]) + q_b[1]) + ... for q_b = q + b stride, b = blockIdx.x.
__global__ void __launch_bounds__(kSeqThreads) k_seq_apply(const float* __restrict__ q, long long stride, long long n,
                                                           const SeqBlock* __restrict__ blocks, int nblocks,
                                                           float* __restrict__ sums) {
    extern __shared__ __align__(16) float seq_buf[];
    __shared__ SeqRun runs[2][32];
    __shared__ float sh_s;
    __shared__ int sh_b;
    q += blockIdx.x * stride;
    blocks += (size_t)blockIdx.x * nblocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh_s = 0.0f;
    int b = 0;
    for (;;) {
        if (warp == 0) {
            __syncwarp();
            float s = sh_s;
            bool ok = true;
            while (ok && b < nblocks) {
                const SeqBlock mine = b + lane < nblocks ? blocks[b + lane] : SeqBlock{seq_identity(), 0u};
                const int m = min(32, nblocks - b);
                int i = 0;
                for (; i < m; ++i) {
                    SeqRun r;
                    r.d = __shfl_sync(0xffffffffu, mine.run.d, i);
                    r.o = __shfl_sync(0xffffffffu, mine.run.o, i);
                    r.mn = __shfl_sync(0xffffffffu, mine.run.mn, i);
                    r.mx = __shfl_sync(0xffffffffu, mine.run.mx, i);
                    ok = seq_apply(s, __shfl_sync(0xffffffffu, mine.binade, i), r);
                    if (!ok) break;
                }
                b += i;
            }
            if (lane == 0) {
                sh_s = s;
                sh_b = b;
            }
        }
        __syncthreads();
        b = sh_b;
        if (b >= nblocks) break;
        // block b by its warps' parts, whose runs are kept for two binades (a sum
        // near a power of two goes back and forth); in any other one warp 0
        // composes the part it needs itself
        seq_stage(seq_buf, q, (long long)b * kSeqBlock, n);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        float t[kSeqTerms];
#pragma unroll
        for (int j = 0; j < kSeqTerms; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(seq_buf + threadIdx.x * kSeqPitch + j);
            t[j] = v.x; t[j + 1] = v.y; t[j + 2] = v.z; t[j + 3] = v.w;
        }
        unsigned have[2] = {0u, 0u};  // binades of runs[0], runs[1]
        int w = 0;                    // parts before w are in the sum
        while (w < 32) {
            const unsigned binade = seq_binade(sh_s);
            if (binade) {
                const int slot = have[0] ? 1 : 0;
                const SeqRun r = seq_warp(seq_run(t, seq_scale(binade)));
                if (lane == 0) runs[slot][warp] = r;
                have[slot] = binade;
            }
            __syncthreads();
            if (warp == 0) {
                float s = sh_s;
                for (; w < 32; ++w) {
                    const unsigned now = seq_binade(s);
                    bool ok = false;
                    if (now == have[0]) {
                        ok = seq_apply(s, now, runs[0][w]);
                    } else if (now == have[1]) {
                        ok = seq_apply(s, now, runs[1][w]);
                    } else if (now && !have[1]) {
                        break;
                    } else if (now) {
                        float u[kSeqTerms];
#pragma unroll
                        for (int j = 0; j < kSeqTerms; j += 4) {
                            const float4 v = *reinterpret_cast<const float4*>(seq_buf + (w * 32 + lane) * kSeqPitch + j);
                            u[j] = v.x; u[j + 1] = v.y; u[j + 2] = v.z; u[j + 3] = v.w;
                        }
                        const SeqRun r = seq_warp(seq_run(u, seq_scale(now)));  // in lane 0
                        if (lane == 0) ok = seq_apply(s, now, r);
                        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                        s = __shfl_sync(0xffffffffu, s, 0);
                    }
                    if (ok) continue;
                    const float4* v = reinterpret_cast<const float4*>(seq_buf + w * 32 * kSeqPitch);
#pragma unroll 4
                    for (int c = 0; c < 32; ++c)
#pragma unroll
                        for (int j = 0; j < kSeqTerms / 4; ++j) {
                            const float4 a = v[c * (kSeqPitch / 4) + j];
                            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
                        }
                }
                if (lane == 0) {
                    sh_s = s;
                    sh_b = w;
                }
            }
            __syncthreads();
            w = sh_b;
        }
        ++b;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = sh_s;
}

}  // namespace gs
