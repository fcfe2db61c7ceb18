// Duplicate merging of picks: gs_merge_duplicates (include/gisspa.h).
//
// Follows the reference's python_scripts/remove_repeat_particles_from_list.py
// (grouping :22-35, visit order :36-50, centre test :53-57, orientation
// distance :59-135, removal rule :136-140).  The pair tests are independent
// and run on the GPU in FP64 (the script's float64): one warp per pick i
// tests the later picks j of its group and lists the duplicate pairs (i, j)
// in j order.  The removal sweep depends on visit order and runs on the host
// over that (sparse) pair list: pick i, if still kept when its turn comes,
// removes each listed j still kept and scoring lower, or is itself removed
// when j scores at least as high, and goes on comparing either way.
#include "gisspa.h"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

namespace {

constexpr double kPiScript = 3.14159265359;  // the script's constant

// What the pair tests need of a pick: its centre, and the cosines and sines of
// its orientation (alt, az, phi), taken once per pick instead of twelve per pair.
struct MergeDev {
    double x, y, ca, sa, cz, sz, cp, sp;
};

__global__ void k_merge_prepare(const gs_merge_item* __restrict__ it, long long n, MergeDev* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const gs_merge_item p = it[i];
    const double alt = p.alt * kPiScript / 180, az = p.az * kPiScript / 180, phi = p.phi * kPiScript / 180;
    out[i] = MergeDev{p.x, p.y, cos(alt), sin(alt), cos(az), sin(az), cos(phi), sin(phi)};
}

// Rotation angle in degrees between two orientations; negative when the script
// skips the pair.
__device__ double euler_distance(const MergeDev& p, const MergeDev& q) {
    const double ca = p.ca, sa = p.sa, cz = p.cz, sz = p.sz, cp = p.cp, sp = p.sp;
    const double cao = q.ca, sao = q.sa, czo = q.cz, szo = q.sz, cpo = q.cp, spo = q.sp;
    double mo[9], m[9], r[9];
    mo[0] = cpo * czo - spo * cao * szo;
    mo[1] = cpo * szo + spo * cao * czo;
    mo[2] = spo * sao;
    mo[3] = -spo * czo - cpo * cao * szo;
    mo[4] = -spo * szo + cpo * cao * czo;
    mo[5] = cpo * sao;
    mo[6] = sao * szo;
    mo[7] = -sao * czo;
    mo[8] = cao;
    m[0] = cp * cz - sp * ca * sz;
    m[1] = -sp * cz - cp * ca * sz;
    m[2] = sa * sz;
    m[3] = cp * sz + sp * ca * cz;
    m[4] = -sp * sz + cp * ca * cz;
    m[5] = -sa * cz;
    m[6] = sp * sa;
    m[7] = cp * sa;
    m[8] = ca;
    r[0] = m[0] * mo[0] + m[3] * mo[1] + m[6] * mo[2];
    r[1] = mo[0] * m[1] + mo[1] * m[4] + mo[2] * m[7];
    r[2] = mo[0] * m[2] + mo[1] * m[5] + mo[2] * m[8];
    r[3] = mo[3] * m[0] + mo[4] * m[3] + mo[5] * m[6];
    r[4] = mo[3] * m[1] + mo[4] * m[4] + mo[5] * m[7];
    r[5] = mo[3] * m[2] + mo[4] * m[5] + mo[5] * m[8];
    r[6] = mo[6] * m[0] + mo[7] * m[3] + mo[8] * m[6];
    r[7] = mo[6] * m[1] + mo[7] * m[4] + mo[8] * m[7];
    r[8] = mo[6] * m[2] + mo[7] * m[5] + mo[8] * m[8];
    const double tr = r[0] + r[4] + r[8];
    double q0 = 0.0;
    if (tr > 0) {
        const double t = sqrt(1 + tr) * 2;
        if (t == 0) return -1.0;
        q0 = 0.25 * t;
    } else {
        // the script's first branch (r0 largest) is evaluated, and may skip the
        // pair, but its q0 is always overridden by the next one
        if (r[0] >= r[4] && r[0] >= r[8]) {
            const double v = 1 + r[0] - r[4] - r[8];
            if (v < 0) return -1.0;  // the script's sqrt would raise here
            if (sqrt(v) * 2 == 0) return -1.0;
        }
        if (r[4] > r[8]) {
            const double v = 1 - r[0] + r[4] - r[8];
            if (v < 0) return -1.0;
            const double t = sqrt(v) * 2;
            if (t == 0) return -1.0;
            q0 = (r[2] - r[6]) / t;
        } else {
            const double v = 1 - r[0] - r[4] + r[8];
            if (v < 0) return -1.0;
            const double t = sqrt(v) * 2;
            if (t == 0) return -1.0;
            q0 = (r[3] - r[1]) / t;
        }
    }
    if (!(q0 <= 1 && q0 >= -1)) return -1.0;
    return fabs(acos(q0) * 2 * 180 / kPiScript);
}

__device__ bool duplicate(const MergeDev& p, const MergeDev& q, double center, double thres) {
    const double dx = q.x - p.x, dy = q.y - p.y;
    const double dist = fabs(sqrt(dx * dx + dy * dy));
    if (!(dist < center)) return false;
    const double ed = euler_distance(p, q);
    if (ed < 0) return false;
    double d2 = fmod(ed, 180.0);
    if (d2 > thres + 1) d2 = 180 - d2;
    return ed < thres || d2 < thres;
}

// Duplicates of every pick i among the later picks of its group, in j order, at
// pairs[off[i] .. off[i] + cnt[i]); total is their number, and where it is
// above cap nothing beyond cap is written.  One warp per i, its lanes
// testing neighbouring j: a thread per i left most of the GPU idle (79 CTAs
// for 20000 picks, 1.5 ms for each of two launches).  Most pairs are far
// apart: `far2`, a little above center^2, settles them without the square root
// and the angles.  The warp keeps the results of its first kMergeKeep steps in
// shared memory, takes its place in the list and writes them out (later
// steps are tested again).  20000 picks in 8 groups: 168 us, against two launches
// of 1.49 ms.
constexpr int kMergeKeep = 128;
__global__ void __launch_bounds__(256) k_merge_pairs(const MergeDev* __restrict__ it, long long n,
                                                     const long long* __restrict__ gend, double center, double thres,
                                                     double far2, unsigned* __restrict__ cnt,
                                                     unsigned long long* __restrict__ off,
                                                     unsigned long long* __restrict__ total, unsigned long long cap,
                                                     unsigned* __restrict__ pairs) {
    __shared__ unsigned keep[8][kMergeKeep];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long i = (long long)blockIdx.x * 8 + warp;
    if (i >= n) return;
    const MergeDev p = it[i];
    const long long end = gend[i];
    const auto step = [&](long long j0) {
        const long long j = j0 + lane;
        bool dup = false;
        if (j < end) {
            const double dx = it[j].x - p.x, dy = it[j].y - p.y;
            if (!(dx * dx + dy * dy > far2)) dup = duplicate(p, it[j], center, thres);
        }
        return __ballot_sync(0xffffffffu, dup);
    };
    unsigned c = 0;
    int k = 0;
    for (long long j0 = i + 1; j0 < end; j0 += 32, ++k) {
        const unsigned m = step(j0);
        if (lane == 0 && k < kMergeKeep) keep[warp][k] = m;
        c += __popc(m);
    }
    unsigned long long o = 0;
    if (lane == 0) {
        if (c) o = atomicAdd(total, (unsigned long long)c);
        cnt[i] = c;
        off[i] = o;
    }
    if (!c) return;
    o = __shfl_sync(0xffffffffu, o, 0);
    __syncwarp();
    k = 0;
    for (long long j0 = i + 1; j0 < end; j0 += 32, ++k) {
        const unsigned m = k < kMergeKeep ? keep[warp][k] : step(j0);
        if (m >> lane & 1u) {
            const unsigned long long at = o + __popc(m & ((1u << lane) - 1u));
            if (at < cap) pairs[at] = (unsigned)(j0 + lane);
        }
        o += __popc(m);
    }
}

struct DevMem {
    void* p = nullptr;
    ~DevMem() { if (p) cudaFree(p); }
};

int cuda_status(cudaError_t e) { return e == cudaSuccess ? GS_OK : GS_ERR_CUDA; }

}  // namespace

extern "C" int gs_merge_duplicates(int device, const gs_merge_item* items, size_t n, double center,
                                   double euler_thres, unsigned char* keep) {
    if ((!items || !keep) && n) return GS_ERR_ARG;
    if (n == 0) return GS_OK;
    if (cudaSetDevice(device) != cudaSuccess) return GS_ERR_CUDA;
    // end of each pick's group (runs of equal group ids)
    std::vector<long long> gend(n);
    for (size_t a = 0; a < n;) {
        size_t b = a;
        while (b < n && items[b].group == items[a].group) ++b;
        for (size_t k = a; k < b; ++k) gend[k] = (long long)b;
        a = b;
    }
    if (n > 0xffffffffull) return GS_ERR_OOM;  // more picks than device memory holds
    // one allocation: items, prepared items, group ends, offsets, total, counts, pairs
    const size_t b_it = sizeof(gs_merge_item) * n, b_ll = sizeof(long long) * n, b_cnt = (sizeof(unsigned) * n + 7) / 8 * 8;
    const size_t b_dev = sizeof(MergeDev) * n, b_in = b_it + b_dev;
    const size_t head = b_in + 2 * b_ll + 8 + b_cnt;
    constexpr unsigned long long kFewPairs = 1024;
    unsigned long long cap = 32ull * n + kFewPairs, total = 0;
    std::vector<unsigned> cnt(n), pairs;
    std::vector<unsigned long long> off(n);
    int st;
    // center^2 with room for the rounding of dx^2 + dy^2 and of the square root
    const double far2 = center * center * (1.0 + 1e-9);
    for (;;) {
        DevMem mem;
        if (cudaMalloc(&mem.p, head + sizeof(unsigned) * cap) != cudaSuccess) {
            cudaGetLastError();
            mem.p = nullptr;
            // not counted yet: without room for pairs first, then for as many as there are
            if (!total && cap > kFewPairs) {
                cap = kFewPairs;
                continue;
            }
            return GS_ERR_OOM;
        }
        char* base = (char*)mem.p;
        gs_merge_item* d_it = (gs_merge_item*)base;
        long long* d_end = (long long*)(base + b_in);
        unsigned long long* d_off = (unsigned long long*)(base + b_in + b_ll);
        unsigned long long* d_total = (unsigned long long*)(base + b_in + 2 * b_ll);
        unsigned* d_cnt = (unsigned*)(base + b_in + 2 * b_ll + 8);
        unsigned* d_pairs = (unsigned*)(base + head);
        if ((st = cuda_status(cudaMemcpy(d_it, items, b_it, cudaMemcpyHostToDevice)))) return st;
        if ((st = cuda_status(cudaMemcpy(d_end, gend.data(), b_ll, cudaMemcpyHostToDevice)))) return st;
        if ((st = cuda_status(cudaMemset(d_total, 0, 8)))) return st;
        MergeDev* d_dev = (MergeDev*)(base + b_it);
        k_merge_prepare<<<(unsigned)((n + 255) / 256), 256>>>(d_it, (long long)n, d_dev);
        k_merge_pairs<<<(unsigned)((n + 7) / 8), 256>>>(d_dev, (long long)n, d_end, center, euler_thres, far2, d_cnt,
                                                         d_off, d_total, cap, d_pairs);
        if ((st = cuda_status(cudaGetLastError()))) return st;
        if ((st = cuda_status(cudaMemcpy(&total, d_total, 8, cudaMemcpyDeviceToHost)))) return st;
        if (total > cap) {  // room for all of them, and again
            cap = total;
            continue;
        }
        pairs.resize(total);
        if ((st = cuda_status(cudaMemcpy(cnt.data(), d_cnt, sizeof(unsigned) * n, cudaMemcpyDeviceToHost)))) return st;
        if ((st = cuda_status(cudaMemcpy(off.data(), d_off, sizeof(unsigned long long) * n, cudaMemcpyDeviceToHost))))
            return st;
        if (total && (st = cuda_status(cudaMemcpy(pairs.data(), d_pairs, sizeof(unsigned) * total, cudaMemcpyDeviceToHost))))
            return st;
        break;
    }
    // the order-dependent removal sweep (:41-49, 136-140)
    std::vector<unsigned char> removed(n, 0);
    for (size_t i = 0; i < n; ++i) {
        if (removed[i]) continue;
        for (unsigned long long k = off[i]; k < off[i] + cnt[i]; ++k) {
            const size_t j = pairs[k];
            if (removed[j]) continue;
            if (items[i].score > items[j].score) removed[j] = 1;
            else removed[i] = 1;
        }
    }
    for (size_t k = 0; k < n; ++k) keep[k] = removed[k] ? 0 : 1;
    return GS_OK;
}
