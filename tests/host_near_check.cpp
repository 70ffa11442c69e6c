// Host check of the meta-cell look-ups of zoom requests: for boxes inside
// another, MetaIndex::among on the outer box's answer gives what
// MetaIndex::query gives, and both what a test of every meta-cell gives.  No
// GPU.
#include "../adeco_gb300/csrc/octree.h"

#include <algorithm>
#include <cstdio>
#include <random>

using namespace adeco;

int main()
{
    std::mt19937_64 rng(8);
    std::uniform_real_distribution<float> U(0.f, 1.f);
    long bad = 0, found = 0;
    for (int grid = 0; grid < 40; ++grid) {
        MetaGrid mg;
        mg.init(20 + (int)(rng() % 60), 20 + (int)(rng() % 60), 20 + (int)(rng() % 60));
        mg.bbox.resize(6 * mg.count());
        const float spread = 5.f * U(rng);
        for (uint64_t id = 0; id < mg.count(); ++id) {
            int org[3], nv[3];
            mg.range(id, org, nv);
            for (int a = 0; a < 3; ++a) {
                mg.bbox[6 * id + a] = (float)org[a] - spread * U(rng);
                mg.bbox[6 * id + 3 + a] = (float)(org[a] + nv[a]) + spread * U(rng);
            }
        }
        MetaIndex index;
        index.build(mg);
        std::vector<uint32_t> near, want, got, all;
        for (int box = 0; box < 50; ++box) {
            float outer[6], inner[6];
            for (int a = 0; a < 3; ++a) {
                outer[a] = 120.f * U(rng) - 20.f;
                outer[3 + a] = outer[a] + 40.f * U(rng) * U(rng);
            }
            index.query(mg, outer, near);
            for (int tile = 0; tile < 20; ++tile) {
                for (int a = 0; a < 3; ++a) {
                    const float x = outer[a] + (outer[3 + a] - outer[a]) * U(rng), y = outer[a] + (outer[3 + a] - outer[a]) * U(rng);
                    const unsigned kind = (unsigned)(rng() % 4);  // faces shared with the outer box, empty boxes
                    inner[a] = kind == 0 ? outer[a] : std::min(x, y);
                    inner[3 + a] = kind == 1 ? outer[3 + a] : (kind == 2 ? inner[a] : std::max(x, y));
                }
                index.query(mg, inner, want);
                MetaIndex::among(mg, near, inner, got);
                all.clear();
                for (uint64_t id = 0; id < mg.count(); ++id) {
                    bool in = true;
                    for (int a = 0; a < 3; ++a) in = in && mg.bbox[6 * id + a] < inner[3 + a] && inner[a] < mg.bbox[6 * id + 3 + a];
                    if (in) all.push_back((uint32_t)id);
                }
                bad += got != want || got != all;
                found += (long)got.size();
            }
        }
    }
    std::printf("%s (%ld found, %ld boxes differ)\n", bad || found < 1000 ? "FAIL" : "ok", found, bad);
    return bad || found < 1000 ? 1 : 0;
}
