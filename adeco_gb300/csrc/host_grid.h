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
