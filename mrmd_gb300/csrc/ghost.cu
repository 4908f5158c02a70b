// Periodic ghost layer: communication::GhostLayer and MultiResGhostLayer.
//
// Ghost creation follows GhostExchange::createGhostAtoms exactly: per axis
// X, Y, Z, every atom (real or earlier ghost) with x < minInner gets an
// image at +L and every atom with x >= maxInner one at -L; images of one
// pass are appended "+L images in source order, then -L images in source
// order", so ghost indices are identical to the reference's.
#include "common.cuh"
#include "ghost_impl.cuh"

using namespace mrmd_impl;

namespace
{
constexpr int TB = 256;

__global__ void k_map_into_domain(double4* __restrict__ pos, int64_t n, double3 mn, double3 mx,
                                  double3 L)
{
    // communication/PeriodicMapping.cpp:30-58
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        double4 p = pos[i];
        double* c[3] = {&p.x, &p.y, &p.z};
        const double mnv[3] = {mn.x, mn.y, mn.z}, mxv[3] = {mx.x, mx.y, mx.z}, Lv[3] = {L.x, L.y, L.z};
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            double x = *c[d];
            if (mxv[d] <= x)
            {
                x = __dsub_rn(x, Lv[d]);
                x = fmax(x, mnv[d]);
            }
            if (x < mnv[d])
            {
                x = __dadd_rn(x, Lv[d]);
                if (mxv[d] <= x) x = mnv[d];
            }
            *c[d] = x;
        }
        pos[i] = p;
    }
}

__device__ __forceinline__ double comp(const double4& p, int axis)
{
    return axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
}

__device__ __forceinline__ void add_comp(double4& p, int axis, double v)
{
    if (axis == 0)
        p.x = __dadd_rn(p.x, v);
    else if (axis == 1)
        p.y = __dadd_rn(p.y, v);
    else
        p.z = __dadd_rn(p.z, v);
}

__device__ __forceinline__ void copy_atom(mrmd_atoms a, int64_t dst, int64_t src)
{
    // data/Atoms.hpp:97-110
    reinterpret_cast<double4*>(a.pos)[dst] = reinterpret_cast<const double4*>(a.pos)[src];
    reinterpret_cast<double4*>(a.vel)[dst] = reinterpret_cast<const double4*>(a.vel)[src];
    reinterpret_cast<double4*>(a.force)[dst] = reinterpret_cast<const double4*>(a.force)[src];
    a.type[dst] = a.type[src];
    a.mass[dst] = a.mass[src];
    a.charge[dst] = a.charge[src];
    a.relativeMass[dst] = a.relativeMass[src];
}

// The ghosts of all three passes from one look at the local items (atoms, or
// molecules in the multi-resolution layer).  An image of a later axis is taken
// of locals and of earlier images alike, and an image keeps its source's
// coordinates on the other axes, so the item's six selection flags
// (x < minInner, x >= maxInner, ...) say which of the 26 images it has.  The
// passes append them kind after kind, each kind in source order: kind k's
// images start where those of the kinds before it end, and an item's place
// among them is the number of items before it that have the kind.
// So: counts per block of items and kind (k_image_count), their scan (one
// block, k_image_scan), the source of every image (k_image_place, for atoms
// with the real atom -> ghosts table: an atom's ghosts ascend with the kind),
// and the copies, one thread an image (k_image_copy, k_image_molecules).
// Three passes of flags, scan, host read-back and copy, then counting,
// scanning, filling and sorting the table, took 26 launches and four round
// trips.  (Copies made by the item's own thread, one kind after the other,
// were bound by the latency of up to 26 copies in a row: 44 us at 32,000
// atoms against 15 for both kernels.)
constexpr int KINDS = 26;
constexpr int IMG_TB = 256;

// flags of kind k: bit 2 d: +L on axis d, bit 2 d + 1: -L.  Atoms take the
// +L images of an axis first, molecules (MOL) the -L ones.
template <bool MOL>
__host__ __device__ constexpr uint32_t kind_flags(int k)
{
    if (MOL) return ((kind_flags<false>(k) & 0x15u) << 1) | ((kind_flags<false>(k) & 0x2au) >> 1);
    if (k < 2) return 1u << k;                                           // x
    const uint32_t xy[3] = {0u, 1u, 2u};
    if (k < 8) return (4u << ((k - 2) / 3)) | xy[(k - 2) % 3];           // y of locals and x images
    const int g = (k - 8) % 9;                                           // z of the nine groups before
    return (16u << ((k - 8) / 9)) | (g < 3 ? xy[g] : ((4u << ((g - 3) / 3)) | xy[(g - 3) % 3]));
}

struct ImageBox
{
    double lo[3], hi[3], L[3];  // inner corners, lengths
};

__device__ __forceinline__ uint32_t image_flags(const double4& p, const ImageBox& b)
{
    uint32_t f = 0u;
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        const double x = comp(p, d);
        f |= (x < b.lo[d] ? 1u : 0u) << (2 * d);
        f |= (x >= b.hi[d] ? 2u : 0u) << (2 * d);
    }
    return f;
}

// rows of counts, one entry per block: images of kind k, and (MOL) their atoms
template <bool MOL>
constexpr int IMG_ROWS = MOL ? 2 * KINDS : KINDS;

// count[row * blocks + block]
template <bool MOL>
__global__ void __launch_bounds__(IMG_TB) k_image_count(const double4* __restrict__ pos,
                                                        const int64_t* __restrict__ numAtoms, int64_t n, ImageBox box,
                                                        int rounds, int32_t* __restrict__ count)
{
    __shared__ int32_t cnt[IMG_ROWS<MOL>];
    if (threadIdx.x < IMG_ROWS<MOL>) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int q = 0; q < rounds; ++q)
    {
        const int64_t i = (blockIdx.x * (int64_t)rounds + q) * IMG_TB + threadIdx.x;
        const uint32_t f = i < n ? image_flags(pos[i], box) : 0u;
        if (__ballot_sync(0xffffffffu, f != 0u) == 0u) continue;
        const int size = MOL && i < n ? (int)numAtoms[i] : 0;
#pragma unroll
        for (int k = 0; k < KINDS; ++k)
        {
            const bool has = (f & kind_flags<MOL>(k)) == kind_flags<MOL>(k);
            const unsigned m = __ballot_sync(0xffffffffu, has);
            if (MOL && m)
            {
                const int atoms = __reduce_add_sync(0xffffffffu, has ? size : 0);
                if ((threadIdx.x & 31) == 0) atomicAdd(&cnt[(MOL ? KINDS : 0) + k], atoms);
            }
            if (m && (threadIdx.x & 31) == 0) atomicAdd(&cnt[k], __popc(m));
        }
    }
    __syncthreads();
    if (threadIdx.x < IMG_ROWS<MOL>) count[threadIdx.x * (int64_t)gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// One warp per kind: exclusive scan over the blocks; then start[k]: images of
// the kinds before k, start[KINDS]: all images; (MOL) KINDS + 1 on, their atoms.
template <bool MOL>
__global__ void __launch_bounds__(KINDS * 32) k_image_scan(int32_t* __restrict__ count, int64_t blocks,
                                                           int64_t* __restrict__ start)
{
    __shared__ int64_t total[IMG_ROWS<MOL>];
    const int lane = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < IMG_ROWS<MOL>; row += KINDS)
    {
        int32_t* c = count + row * blocks;
        int64_t carry = 0;  // (sums of a kind stay below the number of local atoms: 32 bits)
        for (int64_t b0 = 0; b0 < blocks; b0 += 256)
        {
            int32_t v[8], sum = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q)
            {
                const int64_t b = b0 + lane * 8 + q;
                v[q] = b < blocks ? c[b] : 0;
                sum += v[q];
            }
            int32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int32_t off = (int32_t)carry + incl - sum;
#pragma unroll
            for (int q = 0; q < 8; ++q)
            {
                const int64_t b = b0 + lane * 8 + q;
                if (b < blocks) c[b] = off;
                off += v[q];
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) total[row] = carry;
    }
    __syncthreads();
    if (threadIdx.x < (MOL ? 2 : 1))
    {
        int64_t s = 0;
        int64_t* out = start + threadIdx.x * (KINDS + 1);
        for (int q = 0; q < KINDS; ++q)
        {
            out[q] = s;
            s += total[threadIdx.x * KINDS + q];
        }
        out[KINDS] = s;
    }
}

// The source of every image: source[image] (images counted from 0).  Atoms:
// the table ghostStart / ghostList (ghosts counted from n) too.  MOL: atom0,
// the image's first atom (ghost atoms counted from 0).
template <bool MOL>
__global__ void __launch_bounds__(IMG_TB) k_image_place(const double4* __restrict__ pos,
                                                        const int64_t* __restrict__ numAtoms, int64_t n, ImageBox box,
                                                        int rounds, const int32_t* __restrict__ offset,
                                                        const int64_t* __restrict__ start, int64_t limit,
                                                        int32_t* __restrict__ source, int32_t* __restrict__ ghostStart,
                                                        int32_t* __restrict__ ghostList, int32_t* __restrict__ atom0)
{
    constexpr int WARPS = IMG_TB / 32, ROWS = IMG_ROWS<MOL>;
    __shared__ int64_t first[KINDS];
    __shared__ int32_t place[ROWS];           // of the row before this round
    __shared__ int32_t warpCnt[WARPS][ROWS];  // per warp, then exclusive over the warps
    __shared__ int32_t warpImg[WARPS];        // images of the warp's items
    __shared__ int32_t imgBefore;             // images of all items before this round
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    if (threadIdx.x < KINDS) first[threadIdx.x] = start[threadIdx.x];
    if (threadIdx.x < ROWS) place[threadIdx.x] = offset[threadIdx.x * (int64_t)gridDim.x + blockIdx.x];
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int32_t s = 0;
        for (int k = 0; k < KINDS; ++k) s += place[k];
        imgBefore = s;
    }
    for (int q = 0; q < rounds; ++q)
    {
        const int64_t i = (blockIdx.x * (int64_t)rounds + q) * IMG_TB + threadIdx.x;
        const uint32_t f = i < n ? image_flags(pos[i], box) : 0u;
        const int size = MOL && i < n ? (int)numAtoms[i] : 0;
        int32_t mine = 1;  // images of the item
#pragma unroll
        for (int d = 0; d < 3; ++d) mine *= 1 + (int)((f >> (2 * d)) & 1u) + (int)((f >> (2 * d + 1)) & 1u);
        mine -= 1;
        int32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warpImg[warp] = incl;
        const bool any = __ballot_sync(0xffffffffu, f != 0u) != 0u;
        for (int r = lane; r < ROWS; r += 32) warpCnt[warp][r] = 0;
        __syncwarp();
        if (any)
        {
#pragma unroll
            for (int k = 0; k < KINDS; ++k)
            {
                const bool has = (f & kind_flags<MOL>(k)) == kind_flags<MOL>(k);
                const unsigned m = __ballot_sync(0xffffffffu, has);
                if (lane == 0) warpCnt[warp][k] = __popc(m);
                if (MOL && m)
                {
                    const int atoms = __reduce_add_sync(0xffffffffu, has ? size : 0);
                    if (lane == 0) warpCnt[warp][(MOL ? KINDS : 0) + k] = atoms;
                }
            }
        }
        __syncthreads();
        // exclusive over the warps; `place` moves on after the round
        int32_t roundTotal = 0;
        if (threadIdx.x < ROWS)
        {
            for (int w = 0; w < WARPS; ++w)
            {
                const int32_t c = warpCnt[w][threadIdx.x];
                warpCnt[w][threadIdx.x] = place[threadIdx.x] + roundTotal;
                roundTotal += c;
            }
        }
        __syncthreads();
        int32_t list = imgBefore + incl - mine;
        for (int w = 0; w < warp; ++w) list += warpImg[w];
        if (!MOL && i < n) ghostStart[i] = list;
        if (any)
        {
#pragma unroll 2
            for (int k = 0; k < KINDS; ++k)
            {
                const uint32_t kf = kind_flags<MOL>(k);
                const bool has = (f & kf) == kf;
                const unsigned m = __ballot_sync(0xffffffffu, has);
                if (!m) continue;
                int atoms = 0;
                if (MOL)
                {
                    int in = has ? size : 0;
                    atoms = -in;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const int t = __shfl_up_sync(0xffffffffu, in, o);
                        if (lane >= o) in += t;
                    }
                    atoms += in;
                }
                if (!has) continue;
                const int64_t dst = first[k] + warpCnt[warp][k] + __popc(m & below);
                if (!MRMD_IN_BOUNDS(dst, limit)) continue;
                source[dst] = (int32_t)i;
                if (MOL)
                    atom0[dst] = (int32_t)(start[KINDS + 1 + k] + warpCnt[warp][(MOL ? KINDS : 0) + k] + atoms);
                else
                    ghostList[list++] = (int32_t)(n + dst);
            }
        }
        __syncthreads();
        if (threadIdx.x < ROWS) place[threadIdx.x] += roundTotal;
        if (threadIdx.x == 0)
            for (int w = 0; w < WARPS; ++w) imgBefore += warpImg[w];
        __syncthreads();
    }
    if (!MOL && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) ghostStart[n] = (int32_t)start[KINDS];
}

// flags of image g's kind: the kinds' first images are in `start`
template <bool MOL>
__device__ __forceinline__ uint32_t flags_of_image(const int64_t* start, int64_t g)
{
    int k = 0;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1)
        if (k + h < KINDS && start[k + h] <= g) k += h;
    return kind_flags<MOL>(k);
}

// image of a position: the shifts in the order of the axes
__device__ __forceinline__ double4 image_position(double4 p, uint32_t kf, const ImageBox& b)
{
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        if ((kf >> (2 * d)) & 1u) add_comp(p, d, b.L[d]);
        if ((kf >> (2 * d + 1)) & 1u) add_comp(p, d, -b.L[d]);
    }
    return p;
}

__global__ void __launch_bounds__(IMG_TB) k_image_copy(mrmd_atoms a, int64_t n, int64_t nGhost, ImageBox box,
                                                       const int64_t* __restrict__ start,
                                                       const int32_t* __restrict__ corr)
{
    __shared__ int64_t first[KINDS];
    if (threadIdx.x < KINDS) first[threadIdx.x] = start[threadIdx.x];
    __syncthreads();
    const int64_t g = blockIdx.x * (int64_t)IMG_TB + threadIdx.x;
    if (g >= nGhost || !MRMD_IN_BOUNDS(n + g, a.capacity)) return;
    const int64_t src = corr[n + g];
    if (!MRMD_IN_BOUNDS(src, n)) return;
    copy_atom(a, n + g, src);
    double4* pos = reinterpret_cast<double4*>(a.pos);
    pos[n + g] = image_position(pos[src], flags_of_image<false>(first, g), box);
}

// real -> ghosts CSR: count, scan, scatter, then sort each (tiny) segment
__global__ void k_csr_count(const int32_t* __restrict__ corr, int64_t nLocal, int64_t nGhost,
                            int32_t* __restrict__ cnt)
{
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nGhost;
         g += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t r = corr[nLocal + g];
        if (MRMD_IN_BOUNDS(r, nLocal)) atomicAdd(&cnt[r], 1);
    }
}

__global__ void k_csr_fill(const int32_t* __restrict__ corr, int64_t nLocal, int64_t nGhost,
                           const int32_t* __restrict__ start, int32_t* __restrict__ cursor,
                           int32_t* __restrict__ list)
{
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nGhost;
         g += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t r = corr[nLocal + g];
        if (!MRMD_IN_BOUNDS(r, nLocal)) continue;
        const int32_t k = atomicAdd(&cursor[r], 1);
        if (MRMD_IN_BOUNDS(start[r] + k, nGhost)) list[start[r] + k] = (int32_t)(nLocal + g);
    }
}

__global__ void k_csr_sort(const int32_t* __restrict__ start, int64_t nLocal, int32_t* __restrict__ list)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nLocal;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t s = start[i], e = start[i + 1];
        for (int32_t a = s + 1; a < e; ++a)
        {
            int32_t v = list[a];
            int32_t b = a - 1;
            while (b >= s && list[b] > v)
            {
                list[b + 1] = list[b];
                --b;
            }
            list[b + 1] = v;
        }
    }
}

__global__ void k_ghost_update(double4* __restrict__ pos, const int32_t* __restrict__ corr,
                               int64_t nLocal, int64_t nGhost, double3 L, double3 delta)
{
    // communication/UpdateGhostAtoms.cpp:31-68
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < nGhost;
         g += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t idx = nLocal + g;
        if (!MRMD_IN_BOUNDS(corr[idx], nLocal)) continue;
        pos[idx] = ghost_position(pos[idx], pos[corr[idx]], L, delta);
    }
}

template <int AHEAD>
__global__ void k_ghost_reduce(double4* __restrict__ force, const int32_t* __restrict__ start,
                               const int32_t* __restrict__ list, int64_t nLocal, int64_t nGhost)
{
    // communication/AccumulateForce.cpp:25-47, gathered per real atom in
    // ascending ghost order (the serial order of the reference loop).  Bound
    // by its dependent loads in a small system: AHEAD ghosts' entries, then their
    // forces, are loaded at a time (32,000 atoms: 13.2 -> 7.3 us).  A large one
    // has the warps to wait, and four ghosts' registers take half of them away.
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nLocal;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t s = start[i], e = start[i + 1];
        if (s == e) continue;
        double4 f = force[i];
        for (int32_t k0 = s; k0 < e; k0 += AHEAD)
        {
            int32_t g[AHEAD];
            double4 fg[AHEAD];
#pragma unroll
            for (int q = 0; q < AHEAD; ++q)
            {
                g[q] = k0 + q < e ? list[k0 + q] : -1;
                if (g[q] >= 0 && !MRMD_IN_BOUNDS(g[q] - nLocal, nGhost)) g[q] = -1;
            }
#pragma unroll
            for (int q = 0; q < AHEAD; ++q)
                if (g[q] >= 0) fg[q] = force[g[q]];
#pragma unroll
            for (int q = 0; q < AHEAD; ++q)
            {
                if (g[q] < 0) continue;
                f.x = __dadd_rn(f.x, fg[q].x);
                f.y = __dadd_rn(f.y, fg[q].y);
                f.z = __dadd_rn(f.z, fg[q].z);
                force[g[q]] = make_double4(0.0, 0.0, 0.0, 0.0);
            }
        }
        force[i] = f;
    }
}

// ------------------------------------------------------- multi-resolution --

__global__ void k_multires_map(mrmd_molecules m, double4* __restrict__ apos, int64_t nMol,
                               double3 mn, double3 mx, double3 L)
{
    // communication/MultiResRealAtomsExchange.cpp:23-73
    for (int64_t mi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; mi < nMol;
         mi += (int64_t)gridDim.x * blockDim.x)
    {
        double4 p = reinterpret_cast<double4*>(m.pos)[mi];
        const int64_t s = m.atomsOffset[mi], e = s + m.numAtoms[mi];
        const double mnv[3] = {mn.x, mn.y, mn.z}, mxv[3] = {mx.x, mx.y, mx.z}, Lv[3] = {L.x, L.y, L.z};
        for (int d = 0; d < 3; ++d)
        {
            double x = comp(p, d);
            if (mxv[d] <= x)
            {
                x = __dsub_rn(x, Lv[d]);
                for (int64_t a = s; a < e; ++a)
                {
                    double4 q = apos[a];
                    add_comp(q, d, -Lv[d]);
                    apos[a] = q;
                }
            }
            if (x < mnv[d])
            {
                x = __dadd_rn(x, Lv[d]);
                for (int64_t a = s; a < e; ++a)
                {
                    double4 q = apos[a];
                    add_comp(q, d, Lv[d]);
                    apos[a] = q;
                }
            }
            if (d == 0) p.x = x;
            else if (d == 1) p.y = x;
            else p.z = x;
        }
        reinterpret_cast<double4*>(m.pos)[mi] = p;
    }
}

__device__ __forceinline__ void copy_molecule(mrmd_molecules m, int64_t dst, int64_t src)
{
    // data/Molecules.hpp:97-110
    reinterpret_cast<double4*>(m.pos)[dst] = reinterpret_cast<const double4*>(m.pos)[src];
    reinterpret_cast<double4*>(m.force)[dst] = reinterpret_cast<const double4*>(m.force)[src];
    reinterpret_cast<double4*>(m.gradLambda)[dst] = reinterpret_cast<const double4*>(m.gradLambda)[src];
    m.lambda[dst] = m.lambda[src];
    m.modulatedLambda[dst] = m.modulatedLambda[src];
    m.atomsOffset[dst] = m.atomsOffset[src];
    m.numAtoms[dst] = m.numAtoms[src];
}

// Image molecules and their atoms
// (communication/MultiResPeriodicGhostExchange.cpp:147-240).
__global__ void __launch_bounds__(IMG_TB) k_image_molecules(mrmd_molecules m, mrmd_atoms a, int64_t nMol,
                                                            int64_t nAtoms, int64_t nGhost, ImageBox box,
                                                            const int64_t* __restrict__ start,
                                                            const int32_t* __restrict__ source,
                                                            const int32_t* __restrict__ atom0,
                                                            int32_t* __restrict__ corr)
{
    __shared__ int64_t first[KINDS];
    if (threadIdx.x < KINDS) first[threadIdx.x] = start[threadIdx.x];
    __syncthreads();
    const int64_t g = blockIdx.x * (int64_t)IMG_TB + threadIdx.x;
    if (g >= nGhost || !MRMD_IN_BOUNDS(nMol + g, m.capacity)) return;
    const int64_t src = source[g];
    if (!MRMD_IN_BOUNDS(src, nMol)) return;
    const uint32_t kf = flags_of_image<true>(first, g);
    const int64_t s = m.atomsOffset[src], size = m.numAtoms[src], dst = nAtoms + atom0[g];
    copy_molecule(m, nMol + g, src);
    double4* pos = reinterpret_cast<double4*>(m.pos);
    pos[nMol + g] = image_position(pos[src], kf, box);
    m.atomsOffset[nMol + g] = dst;
    pos = reinterpret_cast<double4*>(a.pos);
    for (int64_t k = 0; k < size; ++k)
    {
        if (!MRMD_IN_BOUNDS(dst + k, a.capacity) || !MRMD_IN_BOUNDS(s + k, nAtoms)) break;
        copy_atom(a, dst + k, s + k);
        pos[dst + k] = image_position(pos[s + k], kf, box);
        corr[dst + k] = (int32_t)(s + k);
    }
}

int ensure_layer(mrmd_ctx* ctx, mrmd_ghost_layer* g, int64_t capacity, int64_t localCapacity)
{
    if (capacity > g->capacity)
    {
        int32_t* nc = nullptr;
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&nc), sizeof(int32_t) * (size_t)capacity));
        if (g->correspondingRealAtom && g->capacity > 0)
            MRMD_CUDA(ctx, cudaMemcpyAsync(nc, g->correspondingRealAtom, sizeof(int32_t) * (size_t)g->capacity,
                                           cudaMemcpyDeviceToDevice, ctx->stream));
        int32_t* nl = nullptr;
        if (const int rc = dmalloc(ctx, reinterpret_cast<void**>(&nl), sizeof(int32_t) * (size_t)capacity))
        {
            cudaStreamSynchronize(ctx->stream);
            dfree(nc);
            return rc;
        }
        MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        dfree(g->correspondingRealAtom);
        dfree(g->ghostList);
        g->correspondingRealAtom = nc;
        g->ghostList = nl;
        g->capacity = capacity;
    }
    if (localCapacity > g->localCapacity)
    {
        dfree(g->ghostStart);
        g->ghostStart = nullptr;
        g->localCapacity = g->numLocal = g->numGhost = 0;
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&g->ghostStart), sizeof(int32_t) * (size_t)(localCapacity + 1)));
        g->localCapacity = localCapacity;
    }
    return MRMD_OK;
}

int build_csr(mrmd_ctx* ctx, mrmd_ghost_layer* g, int64_t nLocal, int64_t nGhost)
{
    int32_t* cursor = static_cast<int32_t*>(scratch(ctx, sizeof(int32_t) * (size_t)(nLocal + 1)));
    if (!cursor) return MRMD_ERR_OOM;
    MRMD_CUDA(ctx, cudaMemsetAsync(g->ghostStart, 0, sizeof(int32_t) * (size_t)(nLocal + 1), ctx->stream));
    if (nGhost > 0)
    {
        k_csr_count<<<grid_for(ctx, nGhost, TB), TB, 0, ctx->stream>>>(g->correspondingRealAtom, nLocal,
                                                                        nGhost, g->ghostStart);
        MRMD_TRY(after_launch(ctx, "csr_count"));
    }
    MRMD_TRY(scan_exclusive_i32(ctx, g->ghostStart, g->ghostStart, nLocal + 1, nullptr));
    if (nGhost > 0)
    {
        MRMD_CUDA(ctx, cudaMemsetAsync(cursor, 0, sizeof(int32_t) * (size_t)(nLocal + 1), ctx->stream));
        k_csr_fill<<<grid_for(ctx, nGhost, TB), TB, 0, ctx->stream>>>(
            g->correspondingRealAtom, nLocal, nGhost, g->ghostStart, cursor, g->ghostList);
        MRMD_TRY(after_launch(ctx, "csr_fill"));
        k_csr_sort<<<grid_for(ctx, nLocal, TB), TB, 0, ctx->stream>>>(g->ghostStart, nLocal, g->ghostList);
        MRMD_TRY(after_launch(ctx, "csr_sort"));
    }
    return MRMD_OK;
}

ImageBox image_box(const mrmd_subdomain* sd)
{
    ImageBox box{};
    for (int d = 0; d < 3; ++d)
    {
        box.lo[d] = sd->minInnerCorner[d];
        box.hi[d] = sd->maxInnerCorner[d];
        box.L[d] = sd->diameter[d];
    }
    return box;
}

// Items per block in units of IMG_TB: one for short waits in the blocks, four
// when the one block that scans their counts would take longer than that saves
// (256,000 atoms: count, scan and place 9 + 5 + 22 us with four, 7 + 11 + 14
// with one; 4,000,000: 52 + 37 + 73 with four).
int image_rounds(const mrmd_ctx* ctx, int64_t n) { return n <= (int64_t)ctx->numSMs * 8 * IMG_TB ? 1 : 4; }

inline double3 d3(const double* v) { return make_double3(v[0], v[1], v[2]); }
}  // namespace

extern "C" {

int mrmd_ghost_layer_alloc(mrmd_ctx* ctx, mrmd_ghost_layer* g, int64_t capacity)
{
    if (!ctx || !g) return MRMD_ERR_ARG;
    std::memset(g, 0, sizeof(*g));
    if (capacity < 1) capacity = 1;
    return ensure_layer(ctx, g, capacity, capacity);
}

int mrmd_ghost_layer_free(mrmd_ctx* ctx, mrmd_ghost_layer* g)
{
    if (!g) return MRMD_ERR_ARG;
    if (ctx) cudaStreamSynchronize(ctx->stream);
    dfree(g->correspondingRealAtom);
    dfree(g->ghostStart);
    dfree(g->ghostList);
    std::memset(g, 0, sizeof(*g));
    return MRMD_OK;
}

int mrmd_ghost_exchange_real_atoms(mrmd_ctx* ctx, mrmd_atoms* a, const mrmd_subdomain* sd)
{
    if (!ctx || !a || !sd) return MRMD_ERR_ARG;
    if (a->numLocal == 0) return MRMD_OK;
    k_map_into_domain<<<grid_for(ctx, a->numLocal, TB), TB, 0, ctx->stream>>>(
        reinterpret_cast<double4*>(a->pos), a->numLocal, d3(sd->minCorner), d3(sd->maxCorner),
        d3(sd->diameter));
    MRMD_TRY(after_launch(ctx, "map_into_domain"));
    return finish(ctx, "map_into_domain");
}

int mrmd_ghost_create(mrmd_ctx* ctx, mrmd_ghost_layer* g, mrmd_atoms* a, const mrmd_subdomain* sd)
{
    // GhostExchange::createGhostAtomsXYZ, communication/GhostExchange.cpp:171-181
    if (!ctx || !g || !a || !sd) return MRMD_ERR_ARG;
    const int64_t nLocal = a->numLocal;
    a->numGhost = 0;
    const int rounds = image_rounds(ctx, nLocal);
    const int64_t blocks = div_up(nLocal > 0 ? nLocal : 1, IMG_TB * rounds);
    int64_t* start = static_cast<int64_t*>(
        scratch(ctx, sizeof(int64_t) * (KINDS + 1) + sizeof(int32_t) * KINDS * (size_t)blocks));
    if (!start) return MRMD_ERR_OOM;
    int32_t* counts = reinterpret_cast<int32_t*>(start + KINDS + 1);
    const ImageBox box = image_box(sd);
    const double4* pos = reinterpret_cast<const double4*>(a->pos);
    k_image_count<false><<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(pos, nullptr, nLocal, box, rounds, counts);
    MRMD_TRY(after_launch(ctx, "image_count"));
    k_image_scan<false><<<1, KINDS * 32, 0, ctx->stream>>>(counts, blocks, start);
    MRMD_TRY(after_launch(ctx, "image_scan"));
    int64_t* hTotal = reinterpret_cast<int64_t*>(ctx->hostScalars);
    MRMD_CUDA(ctx, cudaMemcpyAsync(hTotal, start + KINDS, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int64_t nGhost = *hTotal, need = nLocal + nGhost;
    if (need > INT32_MAX) return set_error(ctx, MRMD_ERR_CAPACITY, "more than 2^31 atoms");
    if (need > a->capacity) MRMD_TRY(mrmd_atoms_reserve(ctx, a, need + need / 8 + 64));
    MRMD_TRY(ensure_layer(ctx, g, a->capacity > nLocal + 1 ? a->capacity : nLocal + 1, nLocal + 1));
    // -1: locals and unused entries
    int32_t* corr = g->correspondingRealAtom;
    MRMD_CUDA(ctx, cudaMemsetAsync(corr, 0xff, sizeof(int32_t) * (size_t)g->capacity, ctx->stream));
    k_image_place<false><<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(
        reinterpret_cast<const double4*>(a->pos), nullptr, nLocal, box, rounds, counts, start, nGhost, corr + nLocal,
        g->ghostStart, g->ghostList, nullptr);
    MRMD_TRY(after_launch(ctx, "image_place"));
    if (nGhost > 0)
    {
        k_image_copy<<<(unsigned)div_up(nGhost, IMG_TB), IMG_TB, 0, ctx->stream>>>(*a, nLocal, nGhost, box, start, corr);
        MRMD_TRY(after_launch(ctx, "image_copy"));
    }
    a->numGhost = need - nLocal;
    g->numLocal = a->numLocal;
    g->numGhost = a->numGhost;
    return finish(ctx, "ghost_create");
}

int mrmd_ghost_update(mrmd_ctx* ctx, const mrmd_ghost_layer* g, mrmd_atoms* a, const mrmd_subdomain* sd)
{
    if (!ctx || !g || !a || !sd) return MRMD_ERR_ARG;
    if (g->numLocal != a->numLocal || g->numGhost != a->numGhost)
        return set_error(ctx, MRMD_ERR_STATE, "ghost layer does not match atoms (recreate ghosts)");
    if (a->numGhost == 0) return MRMD_OK;
    const double delta[3] = {0.1 * sd->diameter[0], 0.1 * sd->diameter[1], 0.1 * sd->diameter[2]};
    k_ghost_update<<<grid_for(ctx, a->numGhost, TB), TB, 0, ctx->stream>>>(
        reinterpret_cast<double4*>(a->pos), g->correspondingRealAtom, a->numLocal, a->numGhost,
        d3(sd->diameter), d3(delta));
    MRMD_TRY(after_launch(ctx, "ghost_update"));
    return finish(ctx, "ghost_update");
}

int mrmd_ghost_reduce_force(mrmd_ctx* ctx, const mrmd_ghost_layer* g, mrmd_atoms* a)
{
    if (!ctx || !g || !a) return MRMD_ERR_ARG;
    if (g->numLocal != a->numLocal || g->numGhost != a->numGhost)
        return set_error(ctx, MRMD_ERR_STATE, "ghost layer does not match atoms (recreate ghosts)");
    if (a->numGhost == 0 || a->numLocal == 0) return MRMD_OK;
    auto launch = [&](auto kernel) {
        kernel<<<grid_for(ctx, a->numLocal, TB), TB, 0, ctx->stream>>>(
            reinterpret_cast<double4*>(a->force), g->ghostStart, g->ghostList, a->numLocal, a->numGhost);
    };
    // us of the call with four ghosts ahead / one, fluid in cell order: 4,000
    // atoms 13.6 / 14.0, 32,000 13.5 / 13.3, 128,000 15.8 / 14.8, 1,000,000 25.2
    // / 18.2, 4,000,000 45.4 / 22.8; gas of density 0.02 in random order: 32,000
    // 13.1 / 13.9, 128,000 15.7 / 14.2, 1,000,000 32.5 / 19.8, 4,000,000 73.9 / 31.5
    if (a->numLocal < 400 * (int64_t)ctx->numSMs)
        launch(k_ghost_reduce<4>);
    else
        launch(k_ghost_reduce<1>);
    MRMD_TRY(after_launch(ctx, "ghost_reduce"));
    return finish(ctx, "ghost_reduce");
}

int mrmd_ghost_layer_download(mrmd_ctx* ctx, const mrmd_ghost_layer* g, int64_t n, int64_t* out)
{
    if (!ctx || !g || !out) return MRMD_ERR_ARG;
    MRMD_CHECK_ARG(n >= 0 && n <= g->capacity, ctx, "download size out of range");
    if (n == 0) return MRMD_OK;
    int32_t* tmp = nullptr;
    MRMD_CUDA(ctx, cudaMallocHost(reinterpret_cast<void**>(&tmp), sizeof(int32_t) * (size_t)n));
    cudaError_t e = cudaMemcpyAsync(tmp, g->correspondingRealAtom, sizeof(int32_t) * (size_t)n,
                                    cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess)
        for (int64_t i = 0; i < n; ++i) out[i] = tmp[i];
    cudaFreeHost(tmp);
    return check_cuda(ctx, e, "ghost_layer_download");
}

int mrmd_multires_exchange_real_atoms(mrmd_ctx* ctx, mrmd_molecules* m, mrmd_atoms* a,
                                      const mrmd_subdomain* sd)
{
    if (!ctx || !m || !a || !sd) return MRMD_ERR_ARG;
    if (m->numLocal == 0) return MRMD_OK;
    k_multires_map<<<grid_for(ctx, m->numLocal, TB), TB, 0, ctx->stream>>>(
        *m, reinterpret_cast<double4*>(a->pos), m->numLocal, d3(sd->minCorner), d3(sd->maxCorner),
        d3(sd->diameter));
    MRMD_TRY(after_launch(ctx, "multires_map"));
    return finish(ctx, "multires_map");
}

int mrmd_multires_ghost_create(mrmd_ctx* ctx, mrmd_ghost_layer* g, mrmd_molecules* m, mrmd_atoms* a,
                               const mrmd_subdomain* sd)
{
    // MultiResPeriodicGhostExchange::createGhostAtomsXYZ (:250-265)
    if (!ctx || !g || !m || !a || !sd) return MRMD_ERR_ARG;
    const int64_t nLocal = a->numLocal, nMol = m->numLocal;
    m->numGhost = 0;
    a->numGhost = 0;
    const int rounds = image_rounds(ctx, nMol);
    const int64_t blocks = div_up(nMol > 0 ? nMol : 1, IMG_TB * rounds);
    const size_t head = sizeof(int64_t) * 2 * (KINDS + 1), counted = sizeof(int32_t) * 2 * KINDS * (size_t)blocks;
    auto* mem = static_cast<char*>(scratch(ctx, head + counted));
    if (!mem) return MRMD_ERR_OOM;
    const ImageBox box = image_box(sd);
    k_image_count<true><<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(reinterpret_cast<const double4*>(m->pos),
                                                                      m->numAtoms, nMol, box, rounds,
                                                                      reinterpret_cast<int32_t*>(mem + head));
    MRMD_TRY(after_launch(ctx, "image_count"));
    k_image_scan<true><<<1, KINDS * 32, 0, ctx->stream>>>(reinterpret_cast<int32_t*>(mem + head), blocks,
                                                          reinterpret_cast<int64_t*>(mem));
    MRMD_TRY(after_launch(ctx, "image_scan"));
    int64_t* h = reinterpret_cast<int64_t*>(ctx->hostScalars);
    MRMD_CUDA(ctx, cudaMemcpyAsync(h, mem, head, cudaMemcpyDeviceToHost, ctx->stream));
    MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int64_t addM = h[KINDS], addA = h[2 * KINDS + 1];
    // molecules, atoms and their places among the images are 32-bit indices
    if (nMol + addM > INT32_MAX || nLocal + addA > INT32_MAX)
        return set_error(ctx, MRMD_ERR_CAPACITY, "more than 2^31 molecules or atoms");
    if (nMol + addM > m->capacity) MRMD_TRY(mrmd_molecules_reserve(ctx, m, nMol + addM + (nMol + addM) / 8 + 64));
    if (nLocal + addA > a->capacity)
        MRMD_TRY(mrmd_atoms_reserve(ctx, a, nLocal + addA + (nLocal + addA) / 8 + 64));
    MRMD_TRY(ensure_layer(ctx, g, a->capacity > nLocal + 1 ? a->capacity : nLocal + 1, nLocal + 1));
    MRMD_CUDA(ctx, cudaMemsetAsync(g->correspondingRealAtom, 0xff, sizeof(int32_t) * (size_t)g->capacity, ctx->stream));
    if (addM > 0)
    {
        // sources and first atoms of the images behind the counts (which a
        // larger scratch buffer would lose: they are counted again then)
        const size_t bytes = head + counted + sizeof(int32_t) * 2 * (size_t)addM;
        const bool lost = bytes > ctx->scratchBytes;
        auto* grown = static_cast<char*>(scratch(ctx, bytes));
        if (!grown) return MRMD_ERR_OOM;
        int64_t* start = reinterpret_cast<int64_t*>(grown);
        int32_t* counts = reinterpret_cast<int32_t*>(grown + head);
        if (lost)
        {
            k_image_count<true><<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(
                reinterpret_cast<const double4*>(m->pos), m->numAtoms, nMol, box, rounds, counts);
            MRMD_TRY(after_launch(ctx, "image_count"));
            k_image_scan<true><<<1, KINDS * 32, 0, ctx->stream>>>(counts, blocks, start);
            MRMD_TRY(after_launch(ctx, "image_scan"));
        }
        int32_t* source = counts + 2 * KINDS * blocks;
        k_image_place<true><<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(
            reinterpret_cast<const double4*>(m->pos), m->numAtoms, nMol, box, rounds, counts, start, addM, source,
            nullptr, nullptr, source + addM);
        MRMD_TRY(after_launch(ctx, "image_place"));
        k_image_molecules<<<(unsigned)div_up(addM, IMG_TB), IMG_TB, 0, ctx->stream>>>(
            *m, *a, nMol, nLocal, addM, box, start, source, source + addM, g->correspondingRealAtom);
        MRMD_TRY(after_launch(ctx, "image_molecules"));
    }
    m->numGhost = addM;
    a->numGhost = addA;
    g->numLocal = a->numLocal;
    g->numGhost = a->numGhost;
    MRMD_TRY(build_csr(ctx, g, g->numLocal, g->numGhost));
    return finish(ctx, "multires_ghost_create");
}

}  // extern "C"
