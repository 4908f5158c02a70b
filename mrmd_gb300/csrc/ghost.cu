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

// The ghosts of all three passes from one look at the local atoms.  An
// image of a later axis is taken of locals and of earlier images alike, and an
// image keeps its source's coordinates on the other axes, so the atom's six
// selection flags (x < minInner, x >= maxInner, ...) say which of the 26
// images it has.  The passes append them kind after kind, each kind in source
// order: kind k's images start where those of the kinds before it end, and an
// atom's place among them is the number of atoms before it that have the kind.
// So: counts per block of atoms and kind (k_image_count), their scan (one
// block, k_image_scan), and the images with the real atom -> ghosts table
// (k_image_write); an atom's ghosts ascend with the kind.  (Three passes of
// flags, scan, host read-back and copy, then counting, scanning, filling and
// sorting the table, took 26 launches and four round trips.)
constexpr int KINDS = 26;
constexpr int IMG_TB = 256;
constexpr int IMG_ROUNDS = 4;  // atoms per thread
constexpr int IMG_ATOMS = IMG_TB * IMG_ROUNDS;

// flags of kind k: bit 2 d: +L on axis d, bit 2 d + 1: -L
__host__ __device__ constexpr uint32_t kind_flags(int k)
{
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

// blockCount[k * blocks + block]: atoms of the block with kind k
__global__ void __launch_bounds__(IMG_TB) k_image_count(const double4* __restrict__ pos, int64_t n, ImageBox box,
                                                        int32_t* __restrict__ blockCount)
{
    __shared__ int32_t cnt[KINDS];
    if (threadIdx.x < KINDS) cnt[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < IMG_ROUNDS; ++q)
    {
        const int64_t i = blockIdx.x * (int64_t)IMG_ATOMS + q * IMG_TB + threadIdx.x;
        const uint32_t f = i < n ? image_flags(pos[i], box) : 0u;
        if (__ballot_sync(0xffffffffu, f != 0u) == 0u) continue;
#pragma unroll
        for (int k = 0; k < KINDS; ++k)
        {
            const unsigned m = __ballot_sync(0xffffffffu, (f & kind_flags(k)) == kind_flags(k));
            if (m && (threadIdx.x & 31) == 0) atomicAdd(&cnt[k], __popc(m));
        }
    }
    __syncthreads();
    if (threadIdx.x < KINDS) blockCount[threadIdx.x * (int64_t)gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// One warp per kind: exclusive scan over the blocks; then start[k]: images of
// the kinds before k, start[KINDS]: all images.
__global__ void __launch_bounds__(KINDS * 32) k_image_scan(int32_t* __restrict__ blockCount, int64_t blocks,
                                                           int64_t* __restrict__ start)
{
    __shared__ int64_t total[KINDS];
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    int32_t* c = blockCount + k * blocks;
    int64_t carry = 0;  // (a kind has at most one image per atom: offsets fit 32 bits)
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
    if (lane == 0) total[k] = carry;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int64_t s = 0;
        for (int q = 0; q < KINDS; ++q)
        {
            start[q] = s;
            s += total[q];
        }
        start[KINDS] = s;
    }
}

// The images (data/Atoms.hpp:97-110 with the shifted position), their real
// atoms in corr, and the table ghostStart / ghostList.
__global__ void __launch_bounds__(IMG_TB) k_image_write(mrmd_atoms a, int64_t n, ImageBox box,
                                                        const int32_t* __restrict__ blockOffset,
                                                        const int64_t* __restrict__ start, int32_t* __restrict__ corr,
                                                        int32_t* __restrict__ ghostStart,
                                                        int32_t* __restrict__ ghostList)
{
    constexpr int WARPS = IMG_TB / 32;
    __shared__ int32_t place[KINDS];         // atoms before this round with kind k
    __shared__ int32_t warpCnt[WARPS][KINDS];  // per warp, then exclusive over the warps
    __shared__ int32_t warpImg[WARPS];       // images of the warp's atoms
    __shared__ int32_t imgBefore;            // images of all atoms before this round
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const double4* pos = reinterpret_cast<const double4*>(a.pos);
    if (threadIdx.x < KINDS) place[threadIdx.x] = blockOffset[threadIdx.x * (int64_t)gridDim.x + blockIdx.x];
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int32_t s = 0;
        for (int k = 0; k < KINDS; ++k) s += place[k];
        imgBefore = s;
    }
    for (int q = 0; q < IMG_ROUNDS; ++q)
    {
        const int64_t i = blockIdx.x * (int64_t)IMG_ATOMS + q * IMG_TB + threadIdx.x;
        double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
        if (i < n) p = pos[i];
        const uint32_t f = i < n ? image_flags(p, box) : 0u;
        int32_t mine = 1;  // images of the atom
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
        if (lane < KINDS) warpCnt[warp][lane] = 0;
        __syncwarp();
        if (any)
        {
#pragma unroll
            for (int k = 0; k < KINDS; ++k)
            {
                const unsigned m = __ballot_sync(0xffffffffu, (f & kind_flags(k)) == kind_flags(k));
                if (lane == 0) warpCnt[warp][k] = __popc(m);
            }
        }
        __syncthreads();
        // exclusive over the warps; `place` moves on after the round
        int32_t roundTotal = 0;
        if (threadIdx.x < KINDS)
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
        if (i < n)
        {
            ghostStart[i] = list;
            corr[i] = -1;
        }
        if (any)
        {
#pragma unroll 1
            for (int k = 0; k < KINDS; ++k)
            {
                const uint32_t kf = kind_flags(k);
                const bool has = (f & kf) == kf;
                const unsigned m = __ballot_sync(0xffffffffu, has);
                if (!has) continue;
                const int64_t dst = n + start[k] + warpCnt[warp][k] + __popc(m & below);
                if (!MRMD_IN_BOUNDS(dst, a.capacity)) continue;
                copy_atom(a, dst, i);
                double4 s = p;
#pragma unroll
                for (int d = 0; d < 3; ++d)
                {
                    if ((kf >> (2 * d)) & 1u) add_comp(s, d, box.L[d]);
                    if ((kf >> (2 * d + 1)) & 1u) add_comp(s, d, -box.L[d]);
                }
                reinterpret_cast<double4*>(a.pos)[dst] = s;
                corr[dst] = (int32_t)i;
                ghostList[list++] = (int32_t)dst;
            }
        }
        __syncthreads();
        if (threadIdx.x < KINDS) place[threadIdx.x] += roundTotal;
        if (threadIdx.x == 0)
            for (int w = 0; w < WARPS; ++w) imgBefore += warpImg[w];
        __syncthreads();
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) ghostStart[n] = (int32_t)start[KINDS];
}

__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
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

__global__ void k_ghost_reduce(double4* __restrict__ force, const int32_t* __restrict__ start,
                               const int32_t* __restrict__ list, int64_t nLocal, int64_t nGhost)
{
    // communication/AccumulateForce.cpp:25-47, gathered per real atom in
    // ascending ghost order (the serial order of the reference loop)
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nLocal;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const int32_t s = start[i], e = start[i + 1];
        if (s == e) continue;
        double4 f = force[i];
        for (int32_t k = s; k < e; ++k)
        {
            const int32_t g = list[k];
            if (!MRMD_IN_BOUNDS(g - nLocal, nGhost)) continue;
            const double4 fg = force[g];
            f.x = __dadd_rn(f.x, fg.x);
            f.y = __dadd_rn(f.y, fg.y);
            f.z = __dadd_rn(f.z, fg.z);
            force[g] = make_double4(0.0, 0.0, 0.0, 0.0);
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

// two packed scans: hi = (x >= maxInner: molecules | atoms << 32), lo = (x < minInner)
__global__ void k_multires_flags(mrmd_molecules m, int64_t nMol, int axis, double minInner,
                                 double maxInner, int64_t* __restrict__ hi, int64_t* __restrict__ lo)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nMol;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const double x = comp(reinterpret_cast<const double4*>(m.pos)[i], axis);
        const int64_t na = m.numAtoms[i];
        hi[i] = (x >= maxInner) ? (1 | (na << 32)) : 0;
        lo[i] = (x < minInner) ? (1 | (na << 32)) : 0;
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

__global__ void k_multires_copy(mrmd_molecules m, mrmd_atoms a, int32_t* __restrict__ corr,
                                int64_t nMol, int64_t nAtoms, int axis, double minInner,
                                double maxInner, double L, const int64_t* __restrict__ hiOff,
                                const int64_t* __restrict__ loOff, const int64_t* __restrict__ totals)
{
    // communication/MultiResPeriodicGhostExchange.cpp:147-240: "positive"
    // items (x >= maxInner, shifted by -L) first, then "negative" ones.
    const int64_t posM = totals[0] & 0xffffffffLL, posA = totals[0] >> 32;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nMol;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const double x = comp(reinterpret_cast<const double4*>(m.pos)[i], axis);
        const int64_t s = m.atomsOffset[i], size = m.numAtoms[i];
        for (int side = 0; side < 2; ++side)
        {
            int64_t dstM, dstA;
            double shift;
            if (side == 0)
            {
                if (!(x >= maxInner)) continue;
                dstM = nMol + (hiOff[i] & 0xffffffffLL);
                dstA = nAtoms + (hiOff[i] >> 32);
                shift = -L;
            }
            else
            {
                if (!(x < minInner)) continue;
                dstM = nMol + posM + (loOff[i] & 0xffffffffLL);
                dstA = nAtoms + posA + (loOff[i] >> 32);
                shift = L;
            }
            copy_molecule(m, dstM, i);
            double4 p = reinterpret_cast<double4*>(m.pos)[dstM];
            add_comp(p, axis, shift);
            reinterpret_cast<double4*>(m.pos)[dstM] = p;
            m.atomsOffset[dstM] = dstA;
            m.numAtoms[dstM] = size;
            for (int64_t k = 0; k < size; ++k)
            {
                copy_atom(a, dstA + k, s + k);
                double4 q = reinterpret_cast<double4*>(a.pos)[dstA + k];
                add_comp(q, axis, shift);
                reinterpret_cast<double4*>(a.pos)[dstA + k] = q;
                const int32_t src = (int32_t)(s + k);
                corr[dstA + k] = corr[src] == -1 ? src : corr[src];
            }
        }
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
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&nl), sizeof(int32_t) * (size_t)capacity));
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
    const int64_t blocks = div_up(nLocal > 0 ? nLocal : 1, IMG_ATOMS);
    int64_t* start = static_cast<int64_t*>(
        scratch(ctx, sizeof(int64_t) * (KINDS + 1) + sizeof(int32_t) * KINDS * (size_t)blocks));
    if (!start) return MRMD_ERR_OOM;
    int32_t* counts = reinterpret_cast<int32_t*>(start + KINDS + 1);
    ImageBox box{};
    for (int d = 0; d < 3; ++d)
    {
        box.lo[d] = sd->minInnerCorner[d];
        box.hi[d] = sd->maxInnerCorner[d];
        box.L[d] = sd->diameter[d];
    }
    k_image_count<<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(reinterpret_cast<const double4*>(a->pos), nLocal, box,
                                                                counts);
    MRMD_TRY(after_launch(ctx, "image_count"));
    k_image_scan<<<1, KINDS * 32, 0, ctx->stream>>>(counts, blocks, start);
    MRMD_TRY(after_launch(ctx, "image_scan"));
    int64_t* hTotal = reinterpret_cast<int64_t*>(ctx->hostScalars);
    MRMD_CUDA(ctx, cudaMemcpyAsync(hTotal, start + KINDS, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int64_t need = nLocal + *hTotal;
    if (need > INT32_MAX) return set_error(ctx, MRMD_ERR_CAPACITY, "more than 2^31 atoms");
    if (need > a->capacity) MRMD_TRY(mrmd_atoms_reserve(ctx, a, need + need / 8 + 64));
    MRMD_TRY(ensure_layer(ctx, g, a->capacity > nLocal + 1 ? a->capacity : nLocal + 1, nLocal + 1));
    // -1 (locals and unused entries)
    MRMD_CUDA(ctx, cudaMemsetAsync(g->correspondingRealAtom + need, 0xff, sizeof(int32_t) * (size_t)(g->capacity - need),
                                   ctx->stream));
    k_image_write<<<(unsigned)blocks, IMG_TB, 0, ctx->stream>>>(*a, nLocal, box, counts, start,
                                                                g->correspondingRealAtom, g->ghostStart, g->ghostList);
    MRMD_TRY(after_launch(ctx, "image_write"));
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
    k_ghost_reduce<<<grid_for(ctx, a->numLocal, TB), TB, 0, ctx->stream>>>(
        reinterpret_cast<double4*>(a->force), g->ghostStart, g->ghostList, a->numLocal, a->numGhost);
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
    const int64_t nLocal = a->numLocal;
    MRMD_TRY(ensure_layer(ctx, g, a->capacity > nLocal + 1 ? a->capacity : nLocal + 1, nLocal + 1));
    k_fill_i32<<<grid_for(ctx, g->capacity, TB), TB, 0, ctx->stream>>>(g->correspondingRealAtom,
                                                                        g->capacity, -1);
    MRMD_TRY(after_launch(ctx, "fill_corr"));
    m->numGhost = 0;
    a->numGhost = 0;
    int64_t* totals = reinterpret_cast<int64_t*>(ctx->devScalars);
    for (int axis = 0; axis < 3; ++axis)
    {
        const int64_t nM = m->numLocal + m->numGhost;
        const int64_t nA = a->numLocal + a->numGhost;
        int64_t* hi = static_cast<int64_t*>(scratch(ctx, sizeof(int64_t) * 2 * (size_t)(nM + 1)));
        if (!hi) return MRMD_ERR_OOM;
        int64_t* lo = hi + (nM + 1);
        k_multires_flags<<<grid_for(ctx, nM, TB), TB, 0, ctx->stream>>>(
            *m, nM, axis, sd->minInnerCorner[axis], sd->maxInnerCorner[axis], hi, lo);
        MRMD_TRY(after_launch(ctx, "multires_flags"));
        MRMD_TRY(scan_exclusive_i64(ctx, hi, hi, nM, totals));
        MRMD_TRY(scan_exclusive_i64(ctx, lo, lo, nM, totals + 1));
        int64_t h[2] = {0, 0};
        MRMD_CUDA(ctx, cudaMemcpyAsync(h, totals, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
        MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        const int64_t addM = (h[0] & 0xffffffffLL) + (h[1] & 0xffffffffLL);
        const int64_t addA = (h[0] >> 32) + (h[1] >> 32);
        if (nM + addM > m->capacity) MRMD_TRY(mrmd_molecules_reserve(ctx, m, nM + addM + (nM + addM) / 8 + 64));
        if (nA + addA > a->capacity) MRMD_TRY(mrmd_atoms_reserve(ctx, a, nA + addA + (nA + addA) / 8 + 64));
        MRMD_TRY(ensure_layer(ctx, g, a->capacity, nLocal + 1));
        if (addM > 0)
        {
            k_multires_copy<<<grid_for(ctx, nM, TB), TB, 0, ctx->stream>>>(
                *m, *a, g->correspondingRealAtom, nM, nA, axis, sd->minInnerCorner[axis],
                sd->maxInnerCorner[axis], sd->diameter[axis], hi, lo, totals);
            MRMD_TRY(after_launch(ctx, "multires_copy"));
        }
        m->numGhost += addM;
        a->numGhost += addA;
    }
    g->numLocal = a->numLocal;
    g->numGhost = a->numGhost;
    MRMD_TRY(build_csr(ctx, g, g->numLocal, g->numGhost));
    return finish(ctx, "multires_ghost_create");
}

}  // extern "C"
