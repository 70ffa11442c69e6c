// Host check of a boundary call's sums into the caller's grid (host_grid.h):
// the device adds them only to grids on whole cells, and the host adds a box
// at any address and changes nothing else; the pages of a box's rows are made
// present, no others, and their contents stay.  No GPU.
#include "../adeco_gb300/csrc/host_grid.h"

#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <set>
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

static void rows_touched()
{
    const int dims = 96;  // 3.5 MB of floats: rows of a part of a page
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = sizeof(float) * dims * dims * dims, pages = (bytes + page - 1) / page;
    const int boxes[4][6] = {{0, 0, 0, 96, 96, 96}, {5, 90, 3, 2, 6, 1}, {0, 0, 40, 96, 96, 7}, {95, 95, 95, 1, 1, 1}};
    for (const int *b : boxes) {
        void *m = mmap(nullptr, pages * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (m == MAP_FAILED) {
            ++bad;
            return;
        }
        madvise(m, pages * page, MADV_NOHUGEPAGE);
        touch_rows(m, sizeof(float), dims, b, b + 3, page);
        std::set<size_t> want;
        for (int z = 0; z < b[5]; ++z)
            for (int y = 0; y < b[4]; ++y)
                for (int x = 0; x < b[3]; ++x)
                    want.insert(sizeof(float) * ((size_t)(b[0] + x) + dims * ((size_t)(b[1] + y) + dims * (size_t)(b[2] + z))) / page);
        std::vector<unsigned char> in(pages);
        bad += mincore(m, pages * page, in.data()) != 0;
        for (size_t p = 0; p < pages; ++p) bad += (in[p] & 1) != (want.count(p) != 0);
        munmap(m, pages * page);
    }
    std::vector<float> g(dims * dims * dims);
    for (size_t i = 0; i < g.size(); ++i) g[i] = (float)i;
    touch_rows(g.data(), sizeof(float), dims, boxes[2], boxes[2] + 3, 64);
    for (size_t i = 0; i < g.size(); ++i) bad += g[i] != (float)i;
}

int main()
{
    rows_touched();
    box_at_any_address<float>();
    box_at_any_address<double>();
    std::printf("%s\n", bad ? "FAIL" : "ok");
    return bad ? 1 : 0;
}
