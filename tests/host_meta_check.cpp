// Host check of MetaGrid::cubes on a lattice whose cubes exceed 2^32 (only its
// sizes are needed).  No GPU.
#include "../adeco_gb300/csrc/octree.h"

#include <cstdio>
#include <numeric>
#include <vector>

using namespace adeco;

int main()
{
    int bad = 0;
    const int sizes[3][3] = {{1627, 1627, 1627}, {2000, 1800, 1500}, {16, 9, 8}};
    for (const int *n : sizes) {
        MetaGrid mg;
        mg.init(n[0], n[1], n[2]);
        std::vector<uint32_t> ids(mg.count());
        std::iota(ids.begin(), ids.end(), 0u);
        bad += mg.cubes(ids.data(), ids.size()) != (uint64_t)(n[0] - 1) * (uint64_t)(n[1] - 1) * (uint64_t)(n[2] - 1);
        bad += mg.cubes(ids.data(), 0) != 0;
    }
    std::printf("%s\n", bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
