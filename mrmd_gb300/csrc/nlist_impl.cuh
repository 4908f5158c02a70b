// Cell grid and cell list shared by the list builder, the atom sort and the
// fused stepper.
#pragma once

#include <vector>

#include "common.cuh"
#include "f32_round.cuh"

namespace mrmd_impl
{
struct CellGrid
{
    double3 mn;   // grid origin
    double3 rdx;  // cells per unit length
    int3 n;       // cells per axis
    int64_t ncell;
    double extent;  // max |coordinate| relative bound used for FP32 error bands
    int reach;      // list builds search cells within +-reach per axis
    float3 mnf, rdxf;  // mn, rdx rounded to FP32 (the binning's FP32 estimate)
    float3 h;          // cell edges
    float margin;      // bounds the FP32 rounding of coordinates and cell edges relative to mn
};

// n = max(1, floor(L * reach / delta)) cells per axis, edge L/n >= delta / reach,
// so that every pair within delta is within `reach` cells per axis.
CellGrid make_grid(const double* gridMin, const double* gridMax, double delta, int reach = 1);

// The grid of a half-list build over n particles: cells of half the list
// radius (15 columns of 5 cells hold 174 candidates a row at density 0.8442, 6
// columns of 3 full-radius cells 333: 126 against 155 us at 256,000 atoms),
// unless there would be far more cells than particles (half_radius_cells).  A
// dilute box's rows walk more columns that hold nothing; the whole call is
// shorter there too than it was with full-radius cells and one lane a row: at
// density 0.02 4,000 atoms 57 against 85 us, 256,000 71 against 112, 2,000,000
// 213 against 273, at 0.001 4,000 atoms 53 against 85, 256,000 115 against 157.
CellGrid make_list_grid(const double* gridMin, const double* gridMax, double delta, int64_t n);

// cell = clamp(floor((x - min) * rdx), 0, n - 1) per axis, id (ix*ny + iy)*nz + iz.
// A NaN coordinate goes to cell 0: the comparisons are written so that NaN
// fails `t >= 0` (a double-to-int conversion of NaN is not a valid cell).
// Not inlined: the callers reach it only when the FP32 estimate is open.
static __device__ __noinline__ int32_t cell_coord_fp64(double x, double mn, double rdx, int n)
{
    const double t = floor(__dmul_rn(__dsub_rn(x, mn), rdx));
    int c = t >= 0.0 ? (t > (double)(n - 1) ? n - 1 : (int)t) : 0;
    return c;
}

// The same cell as cell_coord_fp64, from the FP32 estimate where it is
// certain (all but a few in ten thousand coordinates): GB300's FP64 pipe
// made the binning kernel FP64 bound.
__device__ __forceinline__ int32_t cell_coord(double x, double mn, double rdx, int n, float mnf, float rdxf)
{
    bool ok;
    const float t = floor_of_scaled(x, mnf, rdxf, &ok);
    if (!ok) return cell_coord_fp64(x, mn, rdx, n);
    return t >= 0.f ? (t > (float)(n - 1) ? n - 1 : (int)t) : 0;
}

__device__ __forceinline__ int32_t cell_of(const double4& p, const CellGrid& g)
{
    const int32_t cx = cell_coord(p.x, g.mn.x, g.rdx.x, g.n.x, g.mnf.x, g.rdxf.x);
    const int32_t cy = cell_coord(p.y, g.mn.y, g.rdx.y, g.n.y, g.mnf.y, g.rdxf.y);
    const int32_t cz = cell_coord(p.z, g.mn.z, g.rdx.z, g.n.z, g.mnf.z, g.rdxf.z);
    return (cx * g.n.y + cy) * g.n.z + cz;
}

__device__ __forceinline__ bool lex_above(const double4& pi, const double4& pj)
{
    return (pj.x > pi.x) || ((pj.x == pi.x) && ((pj.y > pi.y) || ((pj.y == pi.y) && (pj.z > pi.z))));
}

// The cells of column (ax, ay) that can hold a particle within the list radius
// of the one at (xi, yi, zi) (relative to mn) in cell (cx, cy, .): [z0, z1] cut
// to them; false when there is none.  The distance to a column is that to its
// nearer edge; the outermost cells reach outwards without end, which only adds
// to the far side.  Of the 125 cells within two cells per axis of a sphere of
// two cells' radius 84 remain (half list of 256,000 atoms 133 -> 124 us, tile
// list of 32,000 122 -> 118).
__device__ __forceinline__ bool trim_column(const CellGrid& g, float xi, float yi, float zi, float reachSq, int cx,
                                            int cy, int ax, int ay, int& z0, int& z1)
{
    const float ex = ax > cx ? (float)ax * g.h.x - xi : xi - (float)(ax + 1) * g.h.x;
    const float ey = ay > cy ? (float)ay * g.h.y - yi : yi - (float)(ay + 1) * g.h.y;
    const float dx = ax == cx ? 0.f : fmaxf(ex - g.margin, 0.f), dy = ay == cy ? 0.f : fmaxf(ey - g.margin, 0.f);
    const float rest = __fmaf_rn(-dx, dx, __fmaf_rn(-dy, dy, reachSq));
    if (rest < 0.f) return false;
    float rz;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(rz) : "f"(rest));
    rz = __fmaf_rn(rz, 1.000001f, g.margin);
    z0 = max(z0, min(__float2int_rd((zi - rz) * g.rdxf.z - 1e-3f), g.n.z - 1));
    z1 = min(z1, max(__float2int_rd((zi + rz) * g.rdxf.z + 1e-3f), 0));
    return true;
}

// The candidate spans of particle i in cell ci: the columns within g.reach
// cells per axis (only cell_x >= cell_x(i) for the half list), each column's
// z range [z0, z1] (trim_column) as one contiguous span [s0, s1) of the
// cell-sorted particles.  span(ax, ay, c0, z0, z1, s0, s1) is called in scan
// order (c0: the cell index of (ax, ay, 0)).
template <bool FULL, class Span>
__device__ __forceinline__ void for_each_span(const int32_t* __restrict__ cellStart, const CellGrid& g, int32_t ci,
                                              float xi, float yi, float zi, float reachSq, int64_t nPos, Span&& span,
                                              int part = 0, int parts = 1)
{
    const int cz = ci % g.n.z;
    const int cy = (ci / g.n.z) % g.n.y;
    const int cx = ci / (g.n.z * g.n.y);
    const int R = g.reach;
    const int axEnd = min(cx + R, g.n.x - 1);
    const int za = max(cz - R, 0), zb = min(cz + R, g.n.z - 1);
    const int ay0 = max(cy - R, 0), ay1 = min(cy + R, g.n.y - 1);
    // part `part` of `parts` runs of the columns in scan order
    const int axBegin = FULL ? max(cx - R, 0) : cx, wide = ay1 - ay0 + 1, columns = (axEnd - axBegin + 1) * wide;
    const int first = columns * part / parts, last = columns * (part + 1) / parts;
    for (int ax = axBegin; ax <= axEnd; ++ax)
    {
        for (int ay = ay0; ay <= ay1; ++ay)
        {
            const int column = (ax - axBegin) * wide + ay - ay0;
            if (parts > 1 && (column < first || column >= last)) continue;
            int z0 = za, z1 = zb;
            if (!trim_column(g, xi, yi, zi, reachSq, cx, cy, ax, ay, z0, z1)) continue;
            // cells (ax, ay, z0..z1) are adjacent in the cell order, so their
            // particles form one contiguous span of the sorted arrays
            const int32_t c0 = (ax * g.n.y + ay) * g.n.z;
            const int32_t s0 = cellStart[c0 + z0], s1 = cellStart[c0 + z1 + 1];
            if (!MRMD_IN_BOUNDS(s0, nPos + 1) || !MRMD_IN_BOUNDS(s1, nPos + 1)) continue;
            span(ax, ay, c0, z0, z1, s0, s1);
        }
    }
}

// The candidate test of the list builds: every decision is the FP64
// predicate.  An FP32 prefilter settles the clear cases (outside [rsqLo,
// rsqHi]) and the FP64 positions decide the rest.  FULL: every j != i within
// r; otherwise Cabana's half-neighbour rule (x_j lexicographically above x_i).
// Returns true when j (the candidate q, id in q.w) is kept; d2f: its FP32
// distance squared.
template <bool FULL>
__device__ __forceinline__ bool candidate_kept(const double4* __restrict__ pos, const double4& pi, int64_t i,
                                               float xi, float yi, float zi, const float4& q, double rsq,
                                               float rsqLo, float rsqHi, int64_t nPos, float& d2f)
{
    const int32_t j = __float_as_int(q.w);
    if (j == (int32_t)i || !MRMD_IN_BOUNDS(j, nPos)) return false;
    // lexicographic (x, y, z): float order is exact unless equal
    if (!FULL && q.x < xi) return false;
    const float dx = xi - q.x, dy = yi - q.y, dz = zi - q.z;
    d2f = dx * dx + dy * dy + dz * dz;
    if (d2f > rsqHi) return false;
    if ((FULL || q.x > xi) && d2f < rsqLo) return true;
    const double4 pj = pos[j];
    const double ddx = pi.x - pj.x, ddy = pi.y - pj.y, ddz = pi.z - pj.z;
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
    return (d2 <= rsq) && (FULL || lex_above(pi, pj));
}

// What a list build counts on the device, cleared before it and read back
// with one copy.
struct ListFlags
{
    // longest near and far rows, non-finite position, largest tile, tiles that
    // did not fit, members, tiles with a slice that did not fit
    int32_t i[8];
    unsigned long long totals[2];  // entries of all near and all far rows
};

__host__ __device__ inline unsigned long long* list_totals(int32_t* flags)
{
    return reinterpret_cast<unsigned long long*>(flags + 8);
}

// The warps' entry counts into totals[0] (near or only rows) and [1] (far).
__device__ __forceinline__ void add_totals(uint32_t nearRows, uint32_t farRows,
                                           unsigned long long* __restrict__ totals)
{
    nearRows = __reduce_add_sync(0xffffffffu, nearRows);
    farRows = __reduce_add_sync(0xffffffffu, farRows);
    if ((threadIdx.x & 31) != 0) return;
    if (nearRows) atomicAdd(totals, (unsigned long long)nearRows);
    if (farRows) atomicAdd(totals + 1, (unsigned long long)farRows);
}

// Particles binned by cell: sorted[] holds particle ids in cell order
// (ascending id inside a cell), spos[] their FP32 coordinates relative to
// the grid origin with the id bit-cast into w.
struct CellList
{
    CellGrid g{};
    int32_t* cellOf = nullptr;
    int32_t* cellStart = nullptr;  // [ncell + 1], then the scatter's cursors
    int32_t* unordered = nullptr;
    int32_t* sorted = nullptr;
    float4* spos = nullptr;
    int64_t capN = 0, capCells = 0, numParticles = 0;

    // morton: order the cells along a Z-order curve instead of row-major (for
    // sorting particles; list builds need the row-major order)
    // nonfinite (device, may be null): set to 1 when a position is NaN or
    // infinite; the caller clears it and reads it at its next sync.
    int build(mrmd_ctx* ctx, const double* pos4, int64_t n, const CellGrid& grid, bool morton = false,
              int32_t* nonfinite = nullptr);
    void release();
};

// full = false: Cabana half list; full = true: every j != i within rlist
// (each pair twice, used by the mixed form so that no j-force is scattered).
int build_half_list(mrmd_ctx* ctx, mrmd_nlist* nl, const double* pos4, int64_t nPos, int64_t begin,
                    int64_t end, double rlist, const CellGrid& grid, int64_t maxNeighbors, bool full);
struct TileList;
// Full list split by distance at build time: pairs closer than rnear (FP32
// distance) in nearList, the rest within rlist in farList; the cell list of
// nearList is used.  Each pair appears in exactly one of the two lists.
// With `tiles` (begin = 0), the lists are built in their tile form
// (lj_tile.cuh) only, in one pass (tile_list_launch); when a tile does not
// fit that pass, the int32 rows are built and their tile form made from them.
// onePass = false: always the int32 rows and then their tile form.
int build_split_list(mrmd_ctx* ctx, mrmd_nlist* nearList, mrmd_nlist* farList, const double* pos4, int64_t nPos,
                     int64_t begin, int64_t end, double rlist, double rnear, const CellGrid& grid,
                     TileList* tiles = nullptr, bool onePass = true);
// The tile form of the split full list over rows [0, rows) built in one
// pass from the cell list `cl` (tile_list.cu), without the int32 rows: the
// near/far counts and tl's members and chunks.  flags as build_split_list's;
// flags[4] != 0 when a tile did not fit its tables (the caller then builds
// the int32 rows and their tile form).
int tile_list_launch(mrmd_ctx* ctx, TileList* tl, int64_t rows, int64_t nPos, const CellList& cl, double rsq, float rsqLo, float rsqHi, float nearSqF, mrmd_nlist* nearList,
                     mrmd_nlist* farList, const double* pos4, int32_t* flags);

// MRMD_ERR_ARG unless the list's rows [begin, begin + rows) are particles
// below numLocal and every neighbour index it can hold (the candidates it
// was built over) is below nAll.
int check_list_fits(mrmd_ctx* ctx, const mrmd_nlist* nl, int64_t numLocal, int64_t nAll);
int permute_atoms(mrmd_ctx* ctx, mrmd_atoms* a, mrmd_atoms* shadow, const int32_t* perm, int64_t n);
}  // namespace mrmd_impl
