// The refinement's table of bins (k_ref_maps, refine_weight): which bins are
// selected, and the band-pass factor of the others bit for bit, with the
// cosine edge on both sides of the last selected shell.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "refine.cuh"

using namespace gs;

__global__ void k_weights(const RefineBin* bins, RefineConsts rc, float* weight, int* sel, float* band) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= rc.l * rc.l) return;
    RefinePickDev pk{};
    pk.defocus = 1.5f;
    bool in;
    weight[q] = refine_weight<false>(bins[q], rc, pk, &in, nullptr);
    const int r = shell_index(q % rc.l, q / rc.l, rc.l, rc.l);
    sel[q] = (in ? 1 : 0) | (r >= 0 && r < rc.l / 2 ? 2 : 0);
    band[q] = bandpass<false>(r, rc.hp, rc.lp);
}

int main() {
    int bad = 0;
    for (int l : {32, 96, 300})
        for (float hp : {0.25f * l, 0.5f * l - 7.3f, 0.5f * l - 1.0f, 0.5f * l + 20.0f}) {
            RefineConsts rc{};
            rc.l = l;
            rc.L2 = (long long)l * l;
            rc.apix = 1.0f; rc.lambda = 0.0197f; rc.cs = 2.7f; rc.ampconst = 0.07f;
            rc.kk = 3.0f; rc.a = -9.32f; rc.b = 2.65f; rc.b2 = 0.01908f;
            rc.bf = -78.7757f; rc.bf2 = -12.9121f; rc.bf3 = 1.28732f;
            rc.hp = hp; rc.lp = 0.01f * l; rc.ds = 1.0f / l; rc.d_m = 0.3f * l;
            const int n = l * l;
            char* mem = nullptr;
            if (cudaMalloc(&mem, (size_t)n * (sizeof(RefineBin) + 16)) != cudaSuccess) return 1;
            RefineBin* bins = (RefineBin*)mem;
            float* mask = (float*)(bins + n);
            float *w = mask + n, *b = w + n;
            int* s = (int*)(b + n);
            const int g = (n + 255) / 256;
            k_ref_maps<<<g, 256>>>(mask, bins, rc);
            k_weights<<<g, 256>>>(bins, rc, w, s, b);
            std::vector<float> hw(n), hb(n);
            std::vector<int> hs(n);
            cudaMemcpy(hw.data(), w, 4 * n, cudaMemcpyDeviceToHost);
            cudaMemcpy(hb.data(), b, 4 * n, cudaMemcpyDeviceToHost);
            if (cudaMemcpy(hs.data(), s, 4 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
            cudaFree(mem);
            int wrong = 0, edge = 0;
            for (int q = 0; q < n; ++q) {
                if (hs[q] == 1 || hs[q] == 2) ++wrong;
                if (hs[q] == 0 && memcmp(&hw[q], &hb[q], 4)) ++wrong;
                edge += hs[q] == 0 && hb[q] > 0.0f && hb[q] < 1.0f;
            }
            if (wrong || (hp == 0.5f * l - 1.0f && !edge)) { printf("l %d, hp %g: %d bins wrong (%d on the edge)\n", l, hp, wrong, edge); bad = 1; }
        }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
