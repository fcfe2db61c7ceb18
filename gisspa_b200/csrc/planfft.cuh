// Batched 1D complex FFTs of any length n = A B C held in shared memory, in
// place: with n1 < A, n2 < B, n3 < C and k = k1 + A (k2 + B k3),
//     X[k] = sum_n3 W_C^{n3 k3} [ W_{BC}^{n3 k2} sum_n2 W_B^{n2 k2} [ W_n^{(n2 C + n3) k1}
//            sum_n1 W_A^{n1 k1} x[(n1 B + n2) C + n3] ] ]
// i.e. three register DFTs (regfft.cuh) over one buffer, the result read out
// in digit-reversed places.  Against the mixed-radix Stockham kernel of
// fft.cuh this halves the shared memory (more resident CTAs, wider column
// tiles), takes two or three exchanges instead of one per small radix, has no
// integer division in its loops, and does lengths with a large prime factor
// (the detectors' 3838 = 2 19 101, 3710 = 2 5 7 53 and 4092 = 4 3 11 31) with half the
// multiply-adds of a plain DFT and both operands of most of them in registers.
//
// Bound by latency and issue: three CTAs of 256 threads to an SM (80 registers;
// rows of 5760 values would leave room for four), issue 60 to 63 % over the units of
// window 300 and 36 % where a micrograph's rows make 570 CTAs.  The stage code is one
// function per direction, called by every IO variant of the kernel, so that its
// radices are compiled once.  Twiddles are table entries, of each stage's own table in
// the order that its butterflies read them: from the one table 2 to 5 % of a search
// at windows without kernels of their own, and products of two entries, as fast,
// have up to 6 % more rounding error (512: 1.06e-7 rms, 1.00e-7 with entries; the
// mixed-radix kernel 1.00e-7).
// Without batching, a thread waits for one load at a time (long scoreboard 8 of
// 14 stalled cycles per issue at length 300, 27 % issue): with four in flight and
// 32-bit offsets the 4320 units of 300 x 300 take 5.4 ms instead of 7.5 (4.9 now
// with larger chunks), the preparation of a 4096 x 4096 micrograph 5.0 instead of 6.4
// (eight in flight: the same).
#pragma once

#include "regfft.cuh"

namespace gs {

// n / d for n d < 2^32 (indices into one tile): one multiplication
struct SmallDiv {
    unsigned d, mul;  // mul = ceil(2^32 / d), 0 for d = 1
    static SmallDiv make(unsigned d) { return SmallDiv{d, d == 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d)}; }
};
__device__ __forceinline__ int quot(int n, const SmallDiv& s) { return s.mul ? (int)__umulhi((unsigned)n, s.mul) : n; }

struct PlanDesc {
    int n = 0, A = 0, B = 0, C = 0;  // A = 0: no plan, the Stockham kernel takes it
    int dense = 0;                   // C is a prime without a register DFT
    int P1 = 0, P2 = 0, VP = 0;      // pitches of k1, k2 and of a vector
    SmallDiv dA, dB, dC, dBC, dAC, dAB, dn, dtile;
    const float2* tw = nullptr;      // exp(-2 pi i k / n)
    // the same factors in the order of the stages (plan_tables), or none
    const float2 *twA = nullptr, *twB = nullptr;
};

// The factors of stage A (W_n^{q e} at q B C + e, e < B C) and of stage B
// (W_BC^{q e} at q C + e, e < C) behind one another, so that neighbouring butterflies
// read neighbouring factors: number of them, and the index k of W_n^k that the
// i-th one is.
__host__ __device__ inline int plan_table_size(const PlanDesc& d) {
    return (d.A > 1 && d.B * d.C > 1 ? d.n : 0) + (d.B > 1 && d.C > 1 ? d.B * d.C : 0);
}
__host__ __device__ inline int plan_table_entry(const PlanDesc& d, int i) {
    const int BC = d.B * d.C;
    if (d.A > 1 && BC > 1) {
        if (i < d.n) return (i / BC) * (i % BC);  // below n
        i -= d.n;
    }
    return d.A * (i / d.C) * (i % d.C);
}
inline void plan_tables(PlanDesc* d, const float2* table) {
    d->twA = d->A > 1 && d->B * d->C > 1 ? table : nullptr;
    d->twB = d->B > 1 && d->C > 1 ? table + (d->twA ? d->n : 0) : nullptr;
}

// Register DFTs of the stages.
constexpr bool plan_radix(int r) {
    return r >= 1 && (r <= 20 || r == 23);
}
constexpr int kPlanMaxPrime = 1024;  // of a dense last stage: O(prime) per value

// A B C = n (dense: C prime); false when the Stockham kernel has to do it.
inline bool plan_factors(int n, int* A, int* B, int* C, bool* dense) {
    *dense = false;
    int m = n, big = 0;
    for (int p = 2; (long long)p * p <= m || m > 1;) {
        const bool last = (long long)p * p > m;
        const int f = last ? m : p;
        if (m % f == 0) {
            if (!plan_radix(f)) {
                if (big) return false;
                big = f;
            }
            m /= f;
        } else {
            ++p;
        }
    }
    if (big > kPlanMaxPrime) return false;
    m = big ? n / big : n;
    int best = 1 << 30;
    for (int a = 1; a <= 23; ++a) {
        if (!plan_radix(a) || m % a) continue;
        for (int b = 1; b <= 23; ++b) {
            if (!plan_radix(b) || (m / a) % b) continue;
            const int c = m / a / b;
            if (big ? c != 1 : !plan_radix(c)) continue;
            // fewest stages, then the smallest largest radix; 17, 19 and 23 cost registers
            const int worst = a > b ? (a > c ? a : c) : (b > c ? b : c);
            const int cost = 1000 * ((a > 1) + (b > 1) + (c > 1)) + worst + 2 * (b < a) + (c < b);
            if (cost < best) {
                best = cost;
                *A = a;
                *B = b;
                *C = big ? big : c;
            }
        }
    }
    *dense = big != 0;
    return best < (1 << 30);
}

// Pitches for tiles of `tile` vectors.  P1 and P2 are odd, so that neighbouring
// butterflies of every stage and neighbouring outputs fall into different
// banks; VP, so that a column tile's loads and stores (`tile` vectors by 16 /
// tile elements per half-warp) do.
inline void plan_layout(PlanDesc* d, int tile) {
    d->P2 = d->C | 1;
    d->P1 = (d->B * d->P2) | 1;
    int vp = d->A * d->P1;
    const int want = tile >= 16 ? 1 : tile > 1 ? 16 / tile : 1;
    while (tile >= 16 ? vp % 2 != 1 : vp % 16 != want % 16) ++vp;
    d->VP = vp;
    d->dA = SmallDiv::make(d->A);
    d->dB = SmallDiv::make(d->B);
    d->dC = SmallDiv::make(d->C);
    d->dBC = SmallDiv::make(d->B * d->C);
    d->dAC = SmallDiv::make(d->A * d->C);
    d->dAB = SmallDiv::make(d->A * d->B);
    d->dn = SmallDiv::make(d->n);
    d->dtile = SmallDiv::make(tile);
}

inline size_t plan_smem_bytes(const PlanDesc& d, int tile) {
    return ((size_t)tile * d.VP * (d.dense ? 2 : 1) + (d.dense ? d.C : 0)) * sizeof(float2) +
           (size_t)kFftRedDoubles * sizeof(double);
}

// A tile's offsets fit an int.
inline bool plan_strides_fit(const PlanDesc& d, const VecGeom& g, int tile) {
    return (long long)tile * g.vec_stride + (long long)d.n * g.elem_stride < (1ll << 31);
}

// One stage: per vector `d_count.d` butterflies of radix R; butterfly j starts at
// (j / split) pa + j % split and steps by `stride`.  kTw: output q is multiplied
// by W_n^{q e}, e = tw_mul i, i = tw_low ? j % split : j, a table entry each: the
// stage's own table at q tab_stride + i where there is one, else tw[q e] (these lie
// in up to q cache lines per warp).
struct PlanStage {
    SmallDiv count, split;
    int pa, pb, stride, tw_mul;
    bool tw_low;
    const float2* tab = nullptr;
    int tab_stride = 0;
};

template <int R, bool kInv, bool kTw>
__device__ __forceinline__ void plan_stage(float2* buf, int nv, int VP, const PlanStage& s, const float2* tw) {
    const int total = nv * (int)s.count.d;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int v = quot(t, s.count), j = t - v * (int)s.count.d;
        const int hi = quot(j, s.split), lo = j - hi * (int)s.split.d;
        float2* p = buf + v * VP + hi * s.pa + lo * s.pb;
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = p[q * s.stride];
        if constexpr (R > 1) rf::rfft<R, 1, kInv>(a);
        if constexpr (kTw) {
            const int i = s.tw_low ? lo : j;
            const float2* w = s.tab ? s.tab + i : tw;
            const int step = s.tab ? s.tab_stride : s.tw_mul * i;
            rf::static_for<R>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                constexpr int r = rf::rpos<R>(q);
                p[q * s.stride] = q ? cmul(a[r], twiddle(w, q * step, kInv)) : a[r];
            });
        } else {
            rf::static_for<R>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                p[q * s.stride] = a[rf::rpos<R>(q)];
            });
        }
    }
    __syncthreads();
}

template <bool kInv, bool kTw>
__device__ __forceinline__ void plan_dispatch(int radix, float2* buf, int nv, int VP, const PlanStage& s,
                                              const float2* tw) {
    switch (radix) {
#define GS_PLAN_RADIX(R) case R: plan_stage<R, kInv, kTw>(buf, nv, VP, s, tw); break;
        GS_PLAN_RADIX(2) GS_PLAN_RADIX(3) GS_PLAN_RADIX(4) GS_PLAN_RADIX(5) GS_PLAN_RADIX(6) GS_PLAN_RADIX(7)
        GS_PLAN_RADIX(8) GS_PLAN_RADIX(9) GS_PLAN_RADIX(10) GS_PLAN_RADIX(11) GS_PLAN_RADIX(12) GS_PLAN_RADIX(13)
        GS_PLAN_RADIX(14) GS_PLAN_RADIX(15) GS_PLAN_RADIX(16) GS_PLAN_RADIX(17) GS_PLAN_RADIX(18) GS_PLAN_RADIX(19)
        GS_PLAN_RADIX(20) GS_PLAN_RADIX(23)
#undef GS_PLAN_RADIX
        default: break;
    }
}

// Dense last stage over C (odd prime) contiguous values of every (k1, k2): with
// s_j = a_j + a_{C-j}, d_j = a_j - a_{C-j} the outputs k and C - k are
// (a_0 + sum cos(2 pi jk / C) s_j) -+ i sum sin(2 pi jk / C) d_j.  A thread takes
// one row and kT output pairs; neighbouring threads take neighbouring rows with
// the same outputs, so the cosines are broadcasts.  Result in `alt`.
template <bool kInv>
__device__ __forceinline__ void plan_dense(float2* buf, float2* alt, float2* tab, int nv, const PlanDesc& D) {
    constexpr int kT = 4;
    const int P = D.C, H = (P - 1) / 2, rows = D.A * D.B, step = D.n / P;
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const float2 w = __ldg(D.tw + i * step);
        tab[i] = make_float2(w.x, -w.y);  // (cos, sin)
    }
    const SmallDiv dH = SmallDiv{(unsigned)H, (unsigned)(((1ull << 32) + H - 1) / H)};
    for (int t = threadIdx.x; t < nv * rows * H; t += blockDim.x) {
        const int r = quot(t, dH), j = t - r * H + 1;
        const int v = quot(r, D.dAB), q = r - v * (int)D.dAB.d, k1 = quot(q, D.dB), k2 = q - k1 * D.B;
        float2* a = buf + v * D.VP + k1 * D.P1 + k2 * D.P2;
        const float2 x = a[j], y = a[P - j];
        a[j] = cadd(x, y);
        a[P - j] = csub(x, y);
    }
    __syncthreads();
    const int nr = nv * rows, groups = (H + kT) / kT;  // outputs 0 .. H
    for (int t = threadIdx.x; t < nr * groups; t += blockDim.x) {
        const int g = t / nr, r = t - g * nr;
        const int v = quot(r, D.dAB), q = r - v * (int)D.dAB.d, k1 = quot(q, D.dB), k2 = q - k1 * D.B;
        const int at = v * D.VP + k1 * D.P1 + k2 * D.P2;
        const float2* a = buf + at;
        float2 c[kT], e[kT];
        int idx[kT];
#pragma unroll
        for (int i = 0; i < kT; ++i) {
            c[i] = a[0];
            e[i] = make_float2(0.0f, 0.0f);
            idx[i] = 0;
        }
        for (int j = 1; j <= H; ++j) {
            const float2 s = a[j], d = a[P - j];
#pragma unroll
            for (int i = 0; i < kT; ++i) {
                idx[i] += min(g * kT + i, H);
                if (idx[i] >= P) idx[i] -= P;
                const float2 w = tab[idx[i]];
                c[i] = cfma(s, w.x, c[i]);
                e[i] = cfma(d, w.y, e[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < kT; ++i) {
            const int k = g * kT + i;
            if (k > H) break;
            alt[at + k] = cadd_mi<kInv>(c[i], e[i]);
            if (k) alt[at + P - k] = cadd_mi<!kInv>(c[i], e[i]);
        }
    }
    __syncthreads();
}

// Transforms nv vectors stored element (n1 B + n2) C + n3 at n1 P1 + n2 P2 + n3;
// returns the buffer that holds output k1 + A (k2 + B k3) at k1 P1 + k2 P2 + k3.
template <bool kInv>
static __device__ __noinline__ float2* plan_block_fft(float2* buf, float2* alt, float2* tab, int nv, const PlanDesc& D) {
    const int BC = D.B * D.C;
    if (D.A > 1) {
        PlanStage s{D.dBC, D.dC, D.P2, 1, D.P1, 1, false, D.twA, BC};
        if (BC > 1) plan_dispatch<kInv, true>(D.A, buf, nv, D.VP, s, D.tw);
        else plan_dispatch<kInv, false>(D.A, buf, nv, D.VP, s, D.tw);
    }
    if (D.B > 1) {
        PlanStage s{D.dAC, D.dC, D.P1, 1, D.P2, D.A, true, D.twB, D.C};
        if (D.C > 1) plan_dispatch<kInv, true>(D.B, buf, nv, D.VP, s, D.tw);
        else plan_dispatch<kInv, false>(D.B, buf, nv, D.VP, s, D.tw);
    }
    if (D.dense) {
        plan_dense<kInv>(buf, alt, tab, nv, D);
        return alt;
    }
    if (D.C > 1) {
        PlanStage s{D.dAB, D.dB, D.P1, D.P2, 1, 0, false};
        plan_dispatch<kInv, false>(D.C, buf, nv, D.VP, s, D.tw);
    }
    return buf;
}

// Batched FFT through a plan: the grid, the IO functors and their calls are
// those of fft_batched_kernel.
template <bool kInv, class IO>
__global__ void __launch_bounds__(256, 3) fft_plan_kernel(const __grid_constant__ PlanDesc D, VecGeom g, int tile,
                                                       IO io_param) {
    extern __shared__ float2 smem_plan[];
    IO io = io_param;
    float2* buf = smem_plan;
    float2* alt = smem_plan + (D.dense ? (size_t)tile * D.VP : 0);
    float2* tab = alt + (size_t)tile * D.VP;
    const int img = blockIdx.y;
    const int v0 = blockIdx.x * tile;
    const int nv = min(tile, g.nvec - v0);
    const int n = D.n, tot = nv * n;
    const bool contiguous = g.elem_stride == 1;
    // 32-bit offsets within the tile (plan_strides_fit)
    const long long base = vec_addr(g, img, v0, 0);
    const int vs = (int)g.vec_stride, es = (int)g.elem_stride;
    const SmallDiv dv = nv == tile ? D.dtile : SmallDiv{(unsigned)nv, nv == 1 ? 0u : (0xffffffffu / (unsigned)nv + 1u)};
    // four loads in flight per thread (a clamped index repeats the last load)
    constexpr int kU = 4;
    for (int i0 = threadIdx.x; i0 < tot; i0 += kU * blockDim.x) {
        float2 x[kU];
        int at[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = min(i0 + u * (int)blockDim.x, tot - 1);
            int t, k;
            if (contiguous) { t = quot(i, D.dn); k = i - t * n; }
            else { k = quot(i, dv); t = i - k * nv; }
            const int n1 = quot(k, D.dBC), m = k - n1 * (int)D.dBC.d, n2 = quot(m, D.dC), n3 = m - n2 * D.C;
            at[u] = t * D.VP + n1 * D.P1 + n2 * D.P2 + n3;
            x[u] = io.load(img, v0 + t, k, base + (t * vs + k * es));
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (i0 + u * (int)blockDim.x < tot) buf[at[u]] = x[u];
    }
    __syncthreads();
    const float2* res = plan_block_fft<kInv>(buf, alt, tab, nv, D);
    for (int i = threadIdx.x; i < tot; i += blockDim.x) {
        int t, k;
        if (contiguous) { t = quot(i, D.dn); k = i - t * n; }
        else { k = quot(i, dv); t = i - k * nv; }
        const int q = quot(k, D.dA), k1 = k - q * D.A, k3 = quot(q, D.dB), k2 = q - k3 * D.B;
        io.store(img, v0 + t, k, base + (t * vs + k * es), res[t * D.VP + k1 * D.P1 + k2 * D.P2 + k3]);
    }
    double* red = reinterpret_cast<double*>(smem_plan + (size_t)tile * D.VP * (D.dense ? 2 : 1) + (D.dense ? D.C : 0));
    io.finish(red, v0, nv);
}

}  // namespace gs
