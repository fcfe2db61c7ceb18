// Pixels of the per-pixel maximum (gisspa_b200/csrc/pixmax.cuh): every map
// position falls on its own micrograph pixel or on none, also where the
// micrograph is smaller than the window.
#include <cstdio>
#include <vector>

#include "pixmax.cuh"

using namespace gs;

int main() {
    int bad = 0;
    const int sides[][3] = {{96, 96, 96}, {96, 8, 28}, {96, 95, 300}, {96, 300, 1}, {720, 8, 28}, {300, 301, 299}};
    for (const auto& s : sides) {
        const int l = s[0], nx = s[1], ny = s[2];
        const int offx[2] = {0, nx > l ? nx - l : 0}, offy[2] = {0, ny > l ? ny - l : 0};
        for (int w = 0; w < 4; ++w) {
            std::vector<int> hits((size_t)nx * ny, 0);
            for (int Y = 0; Y < l; ++Y)
                for (int X = 0; X < l; ++X) {
                    const long long at = pixel_of_map(X, Y, offx[w & 1], offy[w >> 1], nx, ny);
                    const int x = offx[w & 1] + X, y = offy[w >> 1] + Y;
                    if (at < 0 ? x < nx && y < ny : at >= (long long)nx * ny || at != (long long)y * nx + x) bad = 1;
                    else if (at >= 0) ++hits[at];
                }
            for (int h : hits) bad |= h > 1;
        }
        if (bad) { printf("window %d, micrograph %d x %d\n", l, nx, ny); break; }
    }
    printf(bad ? "FAIL\n" : "OK\n");
    return bad;
}
