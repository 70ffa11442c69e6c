// Host check of a boundary call's sums into the caller's grid (host_grid.h):
// the device adds them only to grids on whole cells, and the host adds a box
// at any address and changes nothing else.  No GPU.
#include "../adeco_gb300/csrc/host_grid.h"

#include <cstdio>
#include <vector>

using namespace adeco;

static int bad = 0;

template <typename T>
static void box_at_any_address()
{
    const int dims = 5, lo[3] = {1, 0, 2}, ext[3] = {3, 5, 2};
    std::vector<double> packed(3 * 5 * 2);
    for (size_t i = 0; i < packed.size(); ++i) packed[i] = 0.25 * (double)(i + 1);
    for (size_t shift = 0; shift < 2 * sizeof(T); ++shift) {
        alignas(16) char room[sizeof(T) * 125 + 32], want[sizeof room];
        for (size_t i = 0; i < sizeof room; ++i) room[i] = want[i] = (char)(i * 7);
        for (int c = 0; c < 125; ++c) {
            const T v = (T)c;
            std::memcpy(room + shift + sizeof(T) * c, &v, sizeof v);
        }
        std::memcpy(want, room, sizeof room);
        for (int z = 0; z < 2; ++z)
            for (int y = 0; y < 5; ++y)
                for (int x = 0; x < 3; ++x) {
                    const int c = (1 + x) + 5 * (y + 5 * (2 + z));
                    const T v = (T)c + (T)packed[x + 3 * (y + 5 * z)];
                    std::memcpy(want + shift + sizeof(T) * c, &v, sizeof v);
                }
        bad += device_adds(true, room + shift, sizeof(T)) != (shift % sizeof(T) == 0);
        bad += device_adds(false, room + shift, sizeof(T));
        add_box<T>(room + shift, packed.data(), dims, lo, ext);
        bad += std::memcmp(room, want, sizeof room) != 0;
    }
}

int main()
{
    box_at_any_address<float>();
    box_at_any_address<double>();
    std::printf("%s\n", bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
