// Host check of a tet's candidate cells as the mixed kernel takes them, from the
// words of its staged vertices (vertex_range, word_range), against the
// reference's formula for the tet (candidate_range): the same cells, and the
// same answer to whether the tet meets the grid.  Seeded tets over seeded grids
// of 1 to 4096 cells, vertices on cell faces and on the grid's among them, far
// outside, and in planes of constant coordinate.  Built for the host only; no
// GPU.
#include "../adeco_gb300/csrc/kernels.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>

using namespace adeco;

int main()
{
    std::mt19937_64 rng(31);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const int dims_of[] = {1, 2, 3, 16, 33, 128, 1000, 4095, 4096};
    long bad = 0, meet = 0, tets = 0;
    for (int grid = 0; grid < 3000; ++grid) {
        GridDesc g;
        std::memset(&g, 0, sizeof g);
        g.dims = dims_of[grid % 9];
        const double size = std::exp2(40.0 * U(rng) - 20.0), off = (grid % 4 == 0 ? 0.0 : 100.0 * size * (U(rng) - 0.5));
        for (int a = 0; a < 3; ++a) {
            g.gmin[a] = (float)(off + size * U(rng));
            g.gmax[a] = g.gmin[a] + (float)size;
            if (!(g.gmax[a] > g.gmin[a])) g.gmax[a] = std::nextafterf(g.gmin[a], INFINITY);
            g.delta[a] = (g.gmax[a] - g.gmin[a]) / (float)g.dims;
            g.cull_min[a] = g.gmin[a];
            g.cull_max[a] = g.gmax[a];
        }
        for (int t = 0; t < 400; ++t, ++tets) {
            float p[4][3];
            const double wide = std::exp2(-8.0 * U(rng)) * 2.0;
            for (int a = 0; a < 3; ++a) {
                const double at = -1.0 + 3.0 * U(rng);
                for (int q = 0; q < 4; ++q) {
                    double x = g.gmin[a] + size * (at + wide * (U(rng) - 0.5));
                    const unsigned kind = (unsigned)(rng() % 16);
                    if (kind == 0) x = g.gmin[a];
                    if (kind == 1) x = g.gmax[a];
                    if (kind == 2) x = (double)g.gmin[a] + (double)g.delta[a] * (double)(rng() % (unsigned)(g.dims + 1));
                    if (kind == 3 && q) x = p[q - 1][a];
                    if (kind == 4) x = (U(rng) - 0.5) * 1e30;
                    p[q][a] = (float)x;
                }
            }
            const float3 v[4] = {make_float3(p[0][0], p[0][1], p[0][2]), make_float3(p[1][0], p[1][1], p[1][2]),
                                 make_float3(p[2][0], p[2][1], p[2][2]), make_float3(p[3][0], p[3][1], p[3][2])};
            int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
            const bool meets = candidate_range(v, g, lo, hi);
            // the kernel's minima and maxima, a 16-bit half at a time, and its flags
            uint2 mn = vertex_range(p[0], g, false), mx = mn;
            uint32_t flags = mn.y;
            const auto half = [](uint32_t x, uint32_t y, bool least) {
                const uint32_t l = least ? std::min(x & 0xffffu, y & 0xffffu) : std::max(x & 0xffffu, y & 0xffffu);
                const uint32_t h = least ? std::min(x >> 16, y >> 16) : std::max(x >> 16, y >> 16);
                return l | (h << 16);
            };
            for (int q = 1; q < 4; ++q) {
                const uint2 w = vertex_range(p[q], g, false);
                flags |= w.y;
                mn = make_uint2(half(mn.x, w.x, true), half(mn.y, w.y, true));
                mx = make_uint2(half(mx.x, w.x, false), half(mx.y, w.y, false));
            }
            const bool by_flags = (flags & (kBelowMax | kAboveMin)) == (kBelowMax | kAboveMin);
            bad += by_flags != meets;
            if (!meets) continue;
            ++meet;
            for (int a = 0; a < 3; ++a) {
                int l, h;
                word_range(mn, mx, a, g.dims - 1, l, h);
                bad += l != lo[a] || h != hi[a];
            }
        }
    }
    const bool ok = bad == 0 && meet > tets / 10;
    std::printf("candidate ranges of %ld tets (%ld meet their grid): %s (%ld)\n", tets, meet, ok ? "ok" : "FAIL", bad);
    return ok ? 0 : 1;
}
