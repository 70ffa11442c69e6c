// host_grid.h -- a boundary call's sums into the caller's grid in host memory.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>

namespace adeco {

// The device adds the sums into the caller's grid itself where it reaches
// pageable host memory through the host's page tables and the grid lies on
// whole cells: its loads and stores take no other address.
inline bool device_adds(bool host_tables, const void *data, size_t cell)
{
    return host_tables && reinterpret_cast<uintptr_t>(data) % cell == 0;
}

// Makes the pages of rows [lo, lo + ext) of a dims^3 grid of `size`-byte cells
// present and writable without changing them: a byte of each is combined with
// 0, atomically, so that a thread that adds to other cells of the grid
// meanwhile loses nothing.
inline void touch_rows(void *grid, size_t size, int dims, const int lo[3], const int ext[3], size_t page)
{
    char *base = static_cast<char *>(grid), *next = base;
    const size_t d = (size_t)dims;
    const bool whole = (size_t)ext[0] == d && (size_t)ext[1] == d;
    const size_t rows = whole ? 1 : (size_t)ext[1] * ext[2];
    const size_t len = size * (whole ? d * d * (size_t)ext[2] : (size_t)ext[0]);
    for (size_t r = 0; r < rows; ++r) {
        const size_t y = lo[1] + r % ext[1], z = lo[2] + r / ext[1];
        char *a = base + size * ((size_t)lo[0] + d * (y + d * z)), *end = a + len;
        for (char *p = a > next ? a : next; p < end;) {
            __atomic_fetch_or(reinterpret_cast<unsigned char *>(p), (unsigned char)0, __ATOMIC_RELAXED);
            p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) / page + 1) * page);
            next = p;
        }
    }
}

// Adds the cells [lo, lo + ext) of a dims^3 grid, packed x fastest, into a grid
// at any address.
template <typename T>
inline void add_box(void *grid, const double *packed, int dims, const int lo[3], const int ext[3])
{
    const size_t d = (size_t)dims;
    for (int z = 0; z < ext[2]; ++z)
        for (int y = 0; y < ext[1]; ++y) {
            const double *row = packed + (size_t)ext[0] * (y + (size_t)ext[1] * z);
            char *out = static_cast<char *>(grid) +
                        sizeof(T) * ((size_t)lo[0] + d * ((size_t)(lo[1] + y) + d * (size_t)(lo[2] + z)));
            for (int x = 0; x < ext[0]; ++x) {
                T v;
                std::memcpy(&v, out + sizeof(T) * x, sizeof v);
                v += (T)row[x];
                std::memcpy(out + sizeof(T) * x, &v, sizeof v);
            }
        }
}

}  // namespace adeco
