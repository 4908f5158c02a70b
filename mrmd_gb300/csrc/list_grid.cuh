// The cells of a list build: their number, and their size for a half list.
#pragma once

#include <cmath>
#include <cstdint>

namespace mrmd_impl
{
// max(1, floor(L / edge)), at most 2^31 - 1
inline int64_t cells_per_axis(double L, double edge)
{
    const double c = std::floor(L / edge);
    return c >= 2147483647.0 ? 2147483647 : c >= 1.0 ? (int64_t)c : 1;
}

// The cells of a grid, at most 2^48 (three counts of 2^31 would pass 2^63; more
// than 2^31 - 1 cells are refused).
inline int64_t cell_count(int64_t nx, int64_t ny, int64_t nz)
{
    const double cells = (double)nx * (double)ny * (double)nz;
    return cells < 281474976710656.0 ? nx * ny * nz : (int64_t)1 << 48;
}

// True when a half list over n particles is built on cells of half the list
// radius, given the number of those: unless they are far more than the
// particles, or more than their 31-bit indices can number while an eighth of
// them, cells of the full radius, can be.
inline bool half_radius_cells(int64_t cells, int64_t n)
{
    return cells <= 8 * n + 1048576 && cells <= INT32_MAX;
}
}  // namespace mrmd_impl
