// Mixed-form LJ pair force of the fused stepper on shared-memory tiles.
//
// Arithmetic (per pair i, j of the full list, forces written by i only):
// - r^2 as the exact float pair (S + C, err) of lj_tile.cuh.
// - Near rows (pairs closer than r_split + skin/2 at the rebuild) and the rare
//   far-row pair that came closer than r_split: 1/r^2, the LJ force factor
//   u^4 (ff1 u^3 - ff2) and the force products as float pairs (head and
//   first-order error), summed per atom in double-float.
// - Far pairs: one Newton step takes the hardware reciprocal of r^2 to about
//   half an ulp, using the exact low part of r^2; the factor is evaluated in
//   FP32 (|F| <= |F(r_split)| there, 1.16 epsilon/sigma at 1.5 sigma), the
//   forces summed in FP32.
// - Energy and virial: E = ef1 u^6 - ef2 u^3 - shift and -2W = ff1 u^6 - ff2 u^3
//   per uncapped pair (action/LennardJones.hpp:52-78), so the kernel sums
//   u^3, u^6 and the pair count per atom in double-float (these terms are
//   positive: Fast2Sum against a power-of-two offset above any row's sum
//   makes every head addition error-free) and forms E and W once per block
//   in FP64.
//   Capped pairs (inside the capping distance) add their energy and
//   forceFactor * r^2 to separate double-float sums.
// All per-pair work runs on the FP32 pipe: GB300's FP64 rate is a small
// fraction of its FP32 rate, and even the per-atom conversions to FP64 are
// assembled from the float bits with integer operations.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "lj_tile.cuh"
#include "nlist_impl.cuh"

using namespace mrmd_impl;

namespace mrmd_impl
{
bool tile_split_params(const double* origin, double extent, double rlist, SplitParams* out)
{
    int e = 0;
    std::frexp(1.0625 * rlist / 2048.0, &e);  // value in [2^(e-1), 2^e)
    const double Q = std::ldexp(1.0, e);      // smallest power of two above it
    if (!(extent + Q < Q * 16777216.0)) return false;
    *out = make_split(1.0 / Q, Q);
    // the records are differences: any origin on the Q grid serves
    // (split_bits takes it as the integer origin / Q; |origin| < 2^40 Q)
    double o[3];
    for (int d = 0; d < 3; ++d)
    {
        o[d] = std::floor(origin[d] / Q) * Q;
        if (!(std::fabs(o[d]) < Q * 1099511627776.0)) return false;
    }
    out->origin = make_double3(o[0], o[1], o[2]);
    out->ko = make_longlong3((long long)(o[0] / Q), (long long)(o[1] / Q), (long long)(o[2] / Q));
    out->q = -e;  // Q = 2^e
    return true;
}

void TileList::release()
{
    dfree(members);
    dfree(memberCount);
    dfree(nearChunks);
    dfree(farChunks);
    members = memberCount = nullptr;
    nearChunks = farChunks = nullptr;
    tilesCap = nearWords = farWords = tiles = 0;
    nearChunksPerRow = farChunksPerRow = 0;
    maxMembers = 0;
    valid = false;
}

TileParams make_tile_params(const LJDev& p, double rcSqr, double rsplit, int64_t farCapacity)
{
    TileParams t{};
    t.p = p;
    t.rc2 = make_rcsq(rcSqr);
    t.rsplitSq = (float)(rsplit * rsplit);
    // Offsets of the u^3 and u^6 sums: a power of two above the largest sum a
    // row can reach, with its pairs no closer than 0.8 sigma (or the capping
    // distance; sigma^6 = ff1 / (2 ff2)) and up to 2 x the far capacity + 64
    // entries.  A pair closer than that (overlapping atoms without a cap) only
    // loses the error-free property of its own addition.
    const double sig2 = p.ff2 > 0.0 ? std::cbrt(p.ff1 / (2.0 * p.ff2)) : 1.0;
    const double rmin2 = std::fmax(p.capSqr, 0.64 * sig2);
    const double u3max = 1.0 / (rmin2 * rmin2 * rmin2);
    const double n = 2.0 * (double)(farCapacity > 0 ? farCapacity : 64) + 64.0;
    int e3 = 0, e6 = 0;
    std::frexp(n * u3max, &e3);
    std::frexp(n * u3max * u3max, &e6);
    t.bias3 = (float)std::ldexp(1.0, e3);
    t.bias6 = (float)std::ldexp(1.0, e6);
    return t;
}
}  // namespace mrmd_impl

namespace
{
constexpr int HT_BITS = 12;
constexpr int HT = 1 << HT_BITS;  // hash slots per tile (load <= TILE_CAP / HT = 0.75)

__global__ void k_tile_split(const double4* __restrict__ pos, int64_t n, SplitParams sp, float4* __restrict__ rec)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        tile_split(pos[i], sp, rec, i);
}

__device__ __forceinline__ uint32_t slot_hash(int32_t j)
{
    return ((uint32_t)j * 2654435761u) >> (32 - HT_BITS);
}

// The tile form of the split full list just built (k_build_list<1, 1>), one
// block per tile of TILE_ROWS rows.  Phase 1 inserts every neighbour index of
// the rows into a shared open-addressing table of the tile's members, phase 2
// numbers the occupied entries in table order (the member slots), phase 3
// rewrites each row as slots in 8-entry chunks.  flags[3]: largest member
// count; flags[4]: a tile did not fit (its chunks stay unwritten; the pair
// kernel then reads the int32 rows); flags[5]: members of all tiles.
__global__ void __launch_bounds__(TILE_ROWS) k_tile_build(
    const int32_t* __restrict__ countsN, const int32_t* __restrict__ nbrsN, int64_t capN,
    const int32_t* __restrict__ countsF, const int32_t* __restrict__ nbrsF, int64_t capF, int64_t rows, int64_t nAll,
    int32_t* __restrict__ flags, int32_t* __restrict__ members, int32_t* __restrict__ memberCount,
    uint4* __restrict__ nearChunks, int64_t chN, uint4* __restrict__ farChunks, int64_t chF)
{
    extern __shared__ int32_t keys[];                         // [HT]
    uint16_t* slot = reinterpret_cast<uint16_t*>(keys + HT);  // [HT]
    __shared__ int32_t warpTot[TILE_ROWS / 32];
    __shared__ int32_t totalS, badS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t tile = blockIdx.x;
    const int64_t row = tile * TILE_ROWS + tid;
    for (int h = tid; h < HT; h += TILE_ROWS) keys[h] = -1;
    if (tid == 0) badS = 0;
    __syncthreads();

    // most indices are already in the table (a member is the neighbour of
    // about a dozen of the tile's rows): a plain read settles them
    auto insert = [&](int32_t j) {
        if (j < 0 || j >= nAll)
        {
            badS = 1;
            return;
        }
        uint32_t h = slot_hash(j);
        for (int probe = 0; probe < HT; ++probe)
        {
            const int32_t k = keys[h];
            if (k == j) return;
            if (k == -1)
            {
                const int32_t old = atomicCAS(&keys[h], -1, j);
                if (old == -1 || old == j) return;
            }
            h = (h + 1) & (HT - 1);
        }
        badS = 1;  // table full
    };
    int32_t cn = 0, cf = 0;
    const int32_t* colN = nbrsN + mrmd_dev::nbr_row(row, capN);
    const int32_t* colF = nbrsF + mrmd_dev::nbr_row(row, capF);
    if (row < rows)
    {
        cn = countsN[row];
        cf = countsF[row];
        for (int32_t k = 0; k < cn; ++k) insert(colN[32 * (int64_t)k]);
        for (int32_t k = 0; k < cf; ++k) insert(colF[32 * (int64_t)k]);
    }
    __syncthreads();

    // phase 2: slots in table order
    constexpr int PER = HT / TILE_ROWS;
    int32_t local = 0;
    for (int q = 0; q < PER; ++q) local += keys[tid * PER + q] >= 0;
    int32_t incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warpTot[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        int32_t w = lane < TILE_ROWS / 32 ? warpTot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < TILE_ROWS / 32) warpTot[lane] = w;
    }
    __syncthreads();
    int32_t base = (warp > 0 ? warpTot[warp - 1] : 0) + incl - local;
    if (tid == TILE_ROWS - 1) totalS = base + local;
    for (int q = 0; q < PER; ++q)
    {
        const int h = tid * PER + q;
        if (keys[h] >= 0)
        {
            if (base < TILE_CAP)
            {
                slot[h] = (uint16_t)base;
                members[tile * TILE_CAP + base] = keys[h];
            }
            ++base;
        }
    }
    __syncthreads();
    const int32_t total = totalS;
    const bool bad = badS != 0 || total > TILE_CAP;
    if (tid == 0)
    {
        memberCount[tile] = total < TILE_CAP ? total : TILE_CAP;
        atomicMax(&flags[3], total);
        atomicAdd(&flags[5], total);
        if (bad) atomicOr(&flags[4], 1);
    }
    if (bad || row >= rows) return;

    // phase 3: rows as member slots, eight per 16-byte chunk
    auto lookup = [&](int32_t j) -> uint32_t {
        uint32_t h = slot_hash(j);
        for (int probe = 0; probe < HT; ++probe)
        {
            if (keys[h] == j) return slot[h];
            h = (h + 1) & (HT - 1);
        }
        atomicOr(&flags[4], 1);  // unreachable: every kept index was inserted
        return 0u;
    };
    auto write_rows = [&](const int32_t* col, int32_t cnt, uint4* out, int64_t chunks) {
        for (int32_t g0 = 0; g0 < cnt; g0 += 8)
        {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (g0 + q < cnt) w[q >> 1] |= lookup(col[32 * (int64_t)(g0 + q)]) << (16 * (q & 1));
            out[chunk_word(row, g0 >> 3, chunks)] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    };
    write_rows(colN, cn, nearChunks, chN);
    write_rows(colF, cf, farChunks, chF);
}

// ------------------------------------------------------------ pair force --
struct Geom
{
    float dhx, dhy, dhz, dlx, dly, dlz;
    float r2h, r2l;
};

struct Sums
{
    float fxh = 0.f, fxl = 0.f, fyh = 0.f, fyl = 0.f, fzh = 0.f, fzl = 0.f;  // double-float pairs
    float gx = 0.f, gy = 0.f, gz = 0.f;    // FP32 pairs
    float2 sh, sl;                         // biased sums of (u^3, u^6), heads and low parts
    int32_t cnt = 0;                       // uncapped pairs in range
    df ec{0.f, 0.f}, wc{0.f, 0.f};         // capped pairs: energy, forceFactor * r^2
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// The hardware's approximate 1/x alone (__fdividef(1, x) for normal x, without
// its handling of subnormal ones; every use refines or masks it).
__device__ __forceinline__ float rcp_seed(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// s += x for |x| <= bias <= |s| (Fast2Sum: exact error term into the low
// part), u^3 and u^6 side by side
__device__ __forceinline__ void biased_add(float2& sh, float2& sl, float2 x)
{
    const float2 minus = f2(-1.f, -1.f);
    const float2 t = __fadd2_rn(sh, x);
    sl = __fadd2_rn(sl, __ffma2_rn(__ffma2_rn(sh, minus, t), minus, x));  // x - (t - sh)
    sh = t;
}

// s += (dh + dl) * (f0 + f1): FMA TwoProd of the head product, first-order
// cross terms and the TwoSum error into the low part (TwoSum, not an offset
// Fast2Sum: a close contact's pair force can exceed any fixed offset)
__device__ __forceinline__ void acc_prod(float& sh, float& sl, float dh, float dl, float f0, float f1)
{
    const float p = __fmul_rn(dh, f0);
    float e = __fmaf_rn(dh, f0, -p);
    e = __fmaf_rn(dh, f1, __fmaf_rn(dl, f0, e));
    const df t = two_sum(sh, p);
    sl = __fadd_rn(sl, __fadd_rn(e, t.l));
    sh = t.h;
}

template <bool CAP>
__device__ __forceinline__ void near_pair(const Geom& g, const TileParams& tp, Sums& s)
{
    float f0, f1;  // forceFactor = f0 + f1
    if (CAP && g.r2h < tp.p.capSqrf)
    {
        // capped branch (action/LennardJones.hpp:68-72): |F| = capCoeff
        const df r2{g.r2h, g.r2l};
        const df dist = df_sqrt(r2);
        const df ff = df_mul(df{tp.p.capCoeff_f, tp.p.capCoeff_l}, df_rcp(dist));
        f0 = ff.h;
        f1 = ff.l;
        const float e = tp.p.eCapShh - (dist.h - tp.p.capDistf) * tp.p.capCoeff_f;
        df_acc(s.ec, e);
        df_acc(s.wc, ff.h * g.r2h);
    }
    else
    {
        // u = 1/r^2 = u0 + u1 (one Newton step on the exact residual), then
        // u^2, u^3, u^4 and forceFactor = u^4 (ff1 u^3 - ff2) as unnormalised
        // float pairs (head, first-order error)
        const float u0 = rcp_seed(g.r2h);
        const float u1 = __fmul_rn(u0, __fmaf_rn(-g.r2l, u0, __fmaf_rn(-g.r2h, u0, 1.0f)));
        const float p2 = __fmul_rn(u0, u0);
        const float q2 = __fmaf_rn(__fadd_rn(u0, u0), u1, __fmaf_rn(u0, u0, -p2));
        const float p3 = __fmul_rn(p2, u0);
        const float q3 = __fmaf_rn(p2, u1, __fmaf_rn(q2, u0, __fmaf_rn(p2, u0, -p3)));
        const float p4 = __fmul_rn(p2, p2);
        const float q4 = __fmaf_rn(__fadd_rn(p2, p2), q2, __fmaf_rn(p2, p2, -p4));
        const float pa = __fmul_rn(tp.p.ff1h, p3);
        const float qa = __fmaf_rn(tp.p.ff1h, q3, __fmaf_rn(tp.p.ff1l, p3, __fmaf_rn(tp.p.ff1h, p3, -pa)));
        const df ts = two_sum(pa, -tp.p.ff2h);
        const float tl = __fadd_rn(ts.l, __fsub_rn(qa, tp.p.ff2l));
        f0 = __fmul_rn(p4, ts.h);
        f1 = __fmaf_rn(p4, tl, __fmaf_rn(q4, ts.h, __fmaf_rn(p4, ts.h, -f0)));
        // u^3 = p3 + q3 and u^6 = p3^2 + 2 p3 q3 (+ the rounding of p3^2): the
        // head p3 alone carries the seed reciprocal's error, which q3 corrects
        const float u6 = __fmul_rn(p3, p3);
        biased_add(s.sh, s.sl, f2(p3, u6));
        s.sl = __fadd2_rn(s.sl, f2(q3, __fmaf_rn(__fadd_rn(p3, p3), q3, __fmaf_rn(p3, p3, -u6))));
        s.cnt += 1;
    }
    acc_prod(s.fxh, s.fxl, g.dhx, g.dlx, f0, f1);
    acc_prod(s.fyh, s.fyl, g.dhy, g.dly, f0, f1);
    acc_prod(s.fzh, s.fzl, g.dhz, g.dlz, f0, f1);
}

// This row's record with its signs turned, as packed operands.
struct Own
{
    float2 nhxy, nlxy;
    float nhz, nlz;
};

// Two list entries of a row, in their order (has1: the second one exists),
// with the packed FP32 instructions (two lanes per instruction, the rounding
// of the scalar ones): the pair kernel is bound by instruction issue.  x and
// y of a pair share an instruction where each has its own operand; past r^2
// the two pairs share one; u^3 and u^6 of a pair do in the energy sums.  The
// differences are formed as neighbour - own, and r^2 negated, so that no
// packed operand needs a sign change: the products are the same bits.
//   dh = hi_i - hi_j (exact), dl = lo_i - lo_j,
//   S = sum dh^2 (exact), C = sum dl (2 dh + dl), r^2 = S + C as (r2h, r2l);
// the cutoff is decided on the double-float r^2, so that pairs within 2^-24
// of rc^2 land on the same side as in FP64.  Near pairs (NEAR rows, and
// far-row pairs that came within r_split) go to near_pair, the others add
//   u = 1/r^2 (one Newton step), ff = u^4 (ff1 u^3 - ff2)
// (action/LennardJones.hpp:60-66) to the FP32 sums; a pair beyond the
// cutoff, and a near one, takes part with u = 0, which adds exact zeros.
template <bool NEAR, bool CAP>
__device__ __forceinline__ void two_pairs(const Own& o, const float4& a0, const float2& b0, const float4& a1,
                                          const float2& b1, bool has1, const TileParams& tp, Sums& s)
{
    const float2 two = f2(2.f, 2.f), minus = f2(-1.f, -1.f), one = f2(1.f, 1.f);
    const float2 h0 = __fadd2_rn(f2(a0.x, a0.y), o.nhxy), h1 = __fadd2_rn(f2(a1.x, a1.y), o.nhxy);  // -dh x, y
    const float2 l0 = __fadd2_rn(f2(a0.z, a0.w), o.nlxy), l1 = __fadd2_rn(f2(a1.z, a1.w), o.nlxy);  // -dl x, y
    const float2 hz = f2(__fadd_rn(b0.x, o.nhz), __fadd_rn(b1.x, o.nhz));  // -dh z of both pairs
    const float2 lz = f2(__fadd_rn(b0.y, o.nlz), __fadd_rn(b1.y, o.nlz));
    const float2 t0 = __ffma2_rn(two, h0, l0), t1 = __ffma2_rn(two, h1, l1), tz = __ffma2_rn(two, hz, lz);
    const float2 zz = __fmul2_rn(hz, hz), lt = __fmul2_rn(lz, tz);
    const float2 nS = f2(__fmaf_rn(-h0.x, h0.x, __fmaf_rn(-h0.y, h0.y, -zz.x)),
                         __fmaf_rn(-h1.x, h1.x, __fmaf_rn(-h1.y, h1.y, -zz.y)));
    const float2 nC = f2(__fmaf_rn(-l0.x, t0.x, __fmaf_rn(-l0.y, t0.y, -lt.x)),
                         __fmaf_rn(-l1.x, t1.x, __fmaf_rn(-l1.y, t1.y, -lt.y)));
    const float2 nr = __fadd2_rn(nS, nC);                                  // -r2h
    const float2 nq = __ffma2_rn(__ffma2_rn(nS, minus, nr), minus, nC);    // -r2l = -(C - (r2h - S))
    const bool in0 = !(nr.x < -tp.rc2.h || (nr.x == -tp.rc2.h && nq.x < -tp.rc2.l));
    const bool in1 = has1 && !(nr.y < -tp.rc2.h || (nr.y == -tp.rc2.h && nq.y < -tp.rc2.l));
    const bool near0 = in0 && (NEAR || -nr.x < tp.rsplitSq), near1 = in1 && (NEAR || -nr.y < tp.rsplitSq);
    if (NEAR || near0 || near1)
    {
        if (near0) near_pair<CAP>(Geom{-h0.x, -h0.y, -hz.x, -l0.x, -l0.y, -lz.x, -nr.x, -nq.x}, tp, s);
        if (near1) near_pair<CAP>(Geom{-h1.x, -h1.y, -hz.y, -l1.x, -l1.y, -lz.y, -nr.y, -nq.y}, tp, s);
    }
    if (!NEAR)
    {
        float2 u = f2(rcp_seed(-nr.x), rcp_seed(-nr.y));
        u = __ffma2_rn(u, __ffma2_rn(nq, u, __ffma2_rn(nr, u, one)), u);
        const bool far0 = in0 && !near0, far1 = in1 && !near1;
        u = f2(far0 ? u.x : 0.f, far1 ? u.y : 0.f);
        const float2 u2 = __fmul2_rn(u, u), u4 = __fmul2_rn(u2, u2);
        const float c0 = __fmul_rn(u2.x, u.x), c1 = __fmul_rn(u2.y, u.y);  // u^3
        const float f0 = __fmul_rn(u4.x, __fmaf_rn(-tp.p.ff1h, c0, tp.p.ff2h));  // -ff
        const float f1 = __fmul_rn(u4.y, __fmaf_rn(-tp.p.ff1h, c1, tp.p.ff2h));
        const float2 d0 = __fadd2_rn(h0, l0), d1 = __fadd2_rn(h1, l1), dz = __fadd2_rn(hz, lz);
        s.gx = __fmaf_rn(d0.x, f0, s.gx);
        s.gy = __fmaf_rn(d0.y, f0, s.gy);
        s.gz = __fmaf_rn(dz.x, f0, s.gz);
        s.gx = __fmaf_rn(d1.x, f1, s.gx);
        s.gy = __fmaf_rn(d1.y, f1, s.gy);
        s.gz = __fmaf_rn(dz.y, f1, s.gz);
        biased_add(s.sh, s.sl, f2(c0, __fmul_rn(c0, c0)));
        biased_add(s.sh, s.sl, f2(c1, __fmul_rn(c1, c1)));
        s.cnt += (far0 ? 1 : 0) + (far1 ? 1 : 0);
    }
}

// The double with the value of a normal FP32 number (or zero), assembled
// from its bits with integer operations: GB300 runs FP64 conversions on its
// small FP64 pipe.  Subnormal inputs become zero, Inf / NaN keep their class.
__device__ __forceinline__ double f32_as_f64(float x)
{
    const uint32_t b = __float_as_uint(x);
    const uint32_t e = (b >> 23) & 0xffu;
    const uint32_t sign = b & 0x80000000u;
    if (e == 0u) return __hiloint2double((int)sign, 0);
    const uint32_t de = e == 0xffu ? 0x7ffu : e + 896u;
    return __hiloint2double((int)(sign | (de << 20) | ((b >> 3) & 0xfffffu)), (int)(b << 29));
}

// (h + l) as a double: one FP64 addition of two exact conversions
__device__ __forceinline__ double df_as_f64(float h, float l) { return __dadd_rn(f32_as_f64(h), f32_as_f64(l)); }

__device__ __forceinline__ df shfl_down_df(df v, int o)
{
    return df{__shfl_down_sync(0xffffffffu, v.h, o), __shfl_down_sync(0xffffffffu, v.l, o)};
}

// Neighbour records of slot / index `idx`.
template <bool TILE>
__device__ __forceinline__ void load_rec(const float4* __restrict__ shA, const float2* __restrict__ shB,
                                         const float4* __restrict__ rec, int32_t idx, float4& a, float2& b)
{
    if (TILE)
    {
        a = shA[idx];
        b = shB[idx];
    }
    else
    {
        a = __ldg(rec + 2 * (int64_t)idx);
        b = __ldg(reinterpret_cast<const float2*>(rec + 2 * (int64_t)idx + 1));
    }
}

// Asynchronous copies of 16 and 8 bytes from global to shared memory.
__device__ __forceinline__ void async_copy16(void* sh, const void* g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(sh)), "l"(g));
}

__device__ __forceinline__ void async_copy8(void* sh, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(sh)), "l"(g));
}

// TILE: one block per tile, rows as 16-bit member slots in 8-entry chunks
// (capN, capF: chunks per row), member records in shared memory; otherwise
// rows as int32 particle indices (capN, capF: list capacities), records
// gathered from global memory (fallback and comparison form).
//
// No single unit bounds the tiled form: at 256,000 atoms it issues 65% of the
// cycles, the FMA pipe is 46% and the shared-memory pipe 50% busy (the
// neighbours' slots conflict in the banks).  Each row's next chunk is loaded
// before the current one is worked on (957 -> 863 us at 4,000,000 atoms), two
// entries share the packed FP32 instructions (two_pairs), and the records of
// a tile's members arrive by asynchronous copies.  4,000,000 atoms 973 -> 863
// us, 256,000 78 -> 70; of the 863 us the near rows take about 200, the
// staging 70.  128-row tiles stage 28% more members (1068 us).
template <bool TILE, bool CAP>
__global__ void __launch_bounds__(TILE_ROWS, 4) k_lj_tile(
    const float4* __restrict__ rec, const int32_t* __restrict__ members,
    const int32_t* __restrict__ memberCount, int32_t smemStride, const int32_t* __restrict__ countsN,
    const void* __restrict__ colsN, int64_t capN, const int32_t* __restrict__ countsF,
    const void* __restrict__ colsF, int64_t capF, int64_t rows, int64_t nAll, double4* __restrict__ force,
    const TileParams tp, double* __restrict__ ev)
{
    extern __shared__ float4 smem[];
    float4* shA = smem;
    float2* shB = reinterpret_cast<float2*>(smem + smemStride);
    __shared__ float red[TILE_ROWS / 32][10];
    const int tid = threadIdx.x;
    const int64_t tile = blockIdx.x;
    int32_t nMem = 0;
    if (TILE)
    {
        // the members' records: a thread's indices first, then all its copies
        // in flight at once
        constexpr int U = 6;
        nMem = memberCount[tile];
        const int32_t* mem = members + tile * TILE_CAP;
        for (int32_t t0 = tid; t0 < nMem; t0 += U * TILE_ROWS)
        {
            int32_t j[U];
#pragma unroll
            for (int u = 0; u < U; ++u) j[u] = t0 + u * TILE_ROWS < nMem ? __ldg(mem + t0 + u * TILE_ROWS) : -1;
#pragma unroll
            for (int u = 0; u < U; ++u)
            {
                const int32_t t = t0 + u * TILE_ROWS;
                if (t >= nMem || !MRMD_IN_BOUNDS(j[u], nAll)) continue;
                async_copy16(shA + t, rec + 2 * (int64_t)j[u]);
                async_copy8(shB + t, rec + 2 * (int64_t)j[u] + 1);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    const int64_t row = tile * TILE_ROWS + tid;
    const int32_t bound = TILE ? nMem : (int32_t)nAll;
    (void)bound;  // read by MRMD_IN_BOUNDS in the bounds-checked build
    Sums s;
    s.sh = f2(tp.bias3, tp.bias6);
    s.sl = f2(0.f, 0.f);
    if (row < rows)
    {
        float4 ai;
        float2 bi;
        load_rec<false>(nullptr, nullptr, rec, (int32_t)row, ai, bi);
        const int32_t cn = countsN[row], cf = countsF[row];
        const Own own{f2(-ai.x, -ai.y), f2(-ai.z, -ai.w), -bi.x, -bi.y};
        // two entries (slots or particle indices)
        auto pairs = [&](int32_t i0, int32_t i1, bool has1, auto nearRow) {
            if (!MRMD_IN_BOUNDS(i0, bound) || !MRMD_IN_BOUNDS(i1, bound)) return;
            float4 a0, a1;
            float2 b0, b1;
            load_rec<TILE>(shA, shB, rec, i0, a0, b0);
            load_rec<TILE>(shA, shB, rec, i1, a1, b1);
            two_pairs<decltype(nearRow)::value, CAP>(own, a0, b0, a1, b1, has1, tp, s);
        };
        if (TILE)
        {
            // eight slots per 16-byte chunk load, two per word
            auto rows_of = [&](const uint4* __restrict__ chunks, int64_t nch, int32_t cnt, auto nearRow) {
                const uint4* __restrict__ at = chunks + chunk_word(row, 0, nch);
                uint4 next = cnt > 0 ? __ldg(at) : make_uint4(0u, 0u, 0u, 0u);
                for (int32_t left = cnt; left > 0; left -= 8)
                {
                    uint4 c = next;
                    at += 32;
                    if (left > 8) next = __ldg(at);  // in flight while this chunk is worked on
                    for (int32_t m = left < 8 ? left : 8; m > 0; m -= 2)
                    {
                        const int32_t i0 = (int32_t)(c.x & 0xffffu), i1 = m > 1 ? (int32_t)(c.x >> 16) : i0;
                        c.x = c.y;
                        c.y = c.z;
                        c.z = c.w;
                        pairs(i0, i1, m > 1, nearRow);
                    }
                }
            };
            rows_of(static_cast<const uint4*>(colsN), capN, cn, std::true_type{});
            rows_of(static_cast<const uint4*>(colsF), capF, cf, std::false_type{});
        }
        else
        {
            auto rows_of = [&](const int32_t* __restrict__ col, int32_t cnt, auto nearRow) {
                for (int32_t k = 0; k < cnt; k += 2)
                {
                    const int32_t i0 = __ldg(col + 32 * (int64_t)k);
                    const bool has1 = k + 1 < cnt;
                    pairs(i0, has1 ? __ldg(col + 32 * (int64_t)(k + 1)) : i0, has1, nearRow);
                }
            };
            rows_of(static_cast<const int32_t*>(colsN) + mrmd_dev::nbr_row(row, capN), cn, std::true_type{});
            rows_of(static_cast<const int32_t*>(colsF) + mrmd_dev::nbr_row(row, capF), cf, std::false_type{});
        }
        // F = near double-float sum + far FP32 sum
        auto comp = [&](float h, float l, float gsum) -> double {
            const df t = two_sum(h, gsum);
            return df_as_f64(t.h, __fadd_rn(t.l, l));
        };
        force[row] = make_double4(comp(s.fxh, s.fxl, s.gx), comp(s.fyh, s.fyl, s.gy), comp(s.fzh, s.fzl, s.gz), 0.0);
    }
    // per-thread sums without the offsets (exact: the heads lie in
    // [bias, 2 bias)), then a double-float block reduction on the FP32 pipe
    df v[5] = {fast_two_sum(__fsub_rn(s.sh.x, tp.bias3), s.sl.x), fast_two_sum(__fsub_rn(s.sh.y, tp.bias6), s.sl.y),
               df{(float)s.cnt, 0.f}, s.ec, s.wc};
    const int nv = CAP ? 5 : 3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (q < nv) v[q] = df_add(v[q], shfl_down_df(v[q], o));
    const int lane = tid & 31, warp = tid >> 5;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 5; ++q)
        {
            red[warp][2 * q] = v[q].h;
            red[warp][2 * q + 1] = v[q].l;
        }
    __syncthreads();
    if (warp == 0)
    {
#pragma unroll
        for (int q = 0; q < 5; ++q)
            v[q] = lane < TILE_ROWS / 32 ? df{red[lane][2 * q], red[lane][2 * q + 1]} : df{0.f, 0.f};
#pragma unroll
        for (int o = TILE_ROWS / 64; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (q < nv) v[q] = df_add(v[q], shfl_down_df(v[q], o));
        if (lane == 0)
        {
            const double s3 = df_as_f64(v[0].h, v[0].l), s6 = df_as_f64(v[1].h, v[1].l);
            const double c = df_as_f64(v[2].h, v[2].l);
            const double ec = CAP ? df_as_f64(v[3].h, v[3].l) : 0.0, wc = CAP ? df_as_f64(v[4].h, v[4].l) : 0.0;
            // every pair appears in both rows: halve
            const double e = 0.5 * (tp.p.ef1 * s6 - tp.p.ef2 * s3 - tp.p.shift * c + ec);
            const double w = -0.25 * (tp.p.ff1 * s6 - tp.p.ff2 * s3 + wc);
            atomicAdd(ev + 0, e);
            atomicAdd(ev + 1, w);
        }
    }
}
}  // namespace

namespace mrmd_impl
{
int tile_split_coords(mrmd_ctx* ctx, const double* pos4, int64_t n, const SplitParams& sp, float4* rec)
{
    if (n == 0) return MRMD_OK;
    k_tile_split<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(reinterpret_cast<const double4*>(pos4), n, sp, rec);
    return after_launch(ctx, "tile_split");
}

int tile_storage(mrmd_ctx* ctx, TileList* tl, int64_t rows, int64_t capN, int64_t capF)
{
    tl->valid = false;
    tl->tiles = div_up(rows, TILE_ROWS);
    if (tl->tiles > tl->tilesCap)
    {
        dfree(tl->members);
        dfree(tl->memberCount);
        tl->members = tl->memberCount = nullptr;
        tl->tilesCap = 0;
        const int64_t c = tl->tiles + tl->tiles / 8 + 4;
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&tl->members), sizeof(int32_t) * (size_t)c * TILE_CAP));
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&tl->memberCount), sizeof(int32_t) * (size_t)c));
        tl->tilesCap = c;
    }
    tl->nearChunksPerRow = div_up(capN, 8);
    tl->farChunksPerRow = div_up(capF, 8);
    const int64_t rows32 = div_up(rows, 32) * 32;
    if (rows32 * tl->nearChunksPerRow > tl->nearWords)
    {
        dfree(tl->nearChunks);
        tl->nearChunks = nullptr;
        tl->nearWords = 0;
        const int64_t w = rows32 * tl->nearChunksPerRow + rows32 * tl->nearChunksPerRow / 8;
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&tl->nearChunks), sizeof(uint4) * (size_t)w));
        tl->nearWords = w;
    }
    if (rows32 * tl->farChunksPerRow > tl->farWords)
    {
        dfree(tl->farChunks);
        tl->farChunks = nullptr;
        tl->farWords = 0;
        const int64_t w = rows32 * tl->farChunksPerRow + rows32 * tl->farChunksPerRow / 8;
        MRMD_TRY(dmalloc(ctx, reinterpret_cast<void**>(&tl->farChunks), sizeof(uint4) * (size_t)w));
        tl->farWords = w;
    }
    // the pair kernel's shared-memory limit (per device; set here, outside
    // any stream capture)
    const int maxPair = TILE_CAP * (int)(sizeof(float4) + sizeof(float2));
    MRMD_CUDA(ctx, cudaFuncSetAttribute(k_lj_tile<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxPair));
    MRMD_CUDA(ctx, cudaFuncSetAttribute(k_lj_tile<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxPair));
    return MRMD_OK;
}

int tile_build_launch(mrmd_ctx* ctx, TileList* tl, int64_t rows, int64_t nAll, const mrmd_nlist* nearList,
                      const mrmd_nlist* farList, int32_t* flags)
{
    const int64_t capN = nearList->maxNeighbors, capF = farList->maxNeighbors;
    MRMD_TRY(tile_storage(ctx, tl, rows, capN, capF));
    if (rows == 0) return MRMD_OK;
    const size_t smem = sizeof(int32_t) * HT + sizeof(uint16_t) * HT;
    k_tile_build<<<(unsigned)tl->tiles, TILE_ROWS, smem, ctx->stream>>>(
        nearList->counts, nearList->nbrs, capN, farList->counts, farList->nbrs, capF, rows, nAll, flags, tl->members,
        tl->memberCount, tl->nearChunks, tl->nearChunksPerRow, tl->farChunks, tl->farChunksPerRow);
    return after_launch(ctx, "tile_build");
}

void tile_build_done(TileList* tl, int32_t maxMembers, bool valid, int64_t totalMembers)
{
    tl->maxMembers = maxMembers;
    tl->valid = valid;
    tl->totalMembers = totalMembers;
}

int lj_tile_forces(mrmd_ctx* ctx, const TileList* tl, const mrmd_nlist* nearList, const mrmd_nlist* farList,
                   const float4* rec, double* force4, const TileParams& tp, double* ev,
                   int64_t nAll, bool gather)
{
    const int64_t rows = nearList->rows;
    if (rows == 0) return MRMD_OK;
    const unsigned grid = (unsigned)div_up(rows, TILE_ROWS);
    const bool cap = tp.p.capSqr > 0.0;
    double4* f = reinterpret_cast<double4*>(force4);
    if (tl && tl->valid && !gather)
    {
        // members of the largest tile, rounded to 16 (shB starts 16-byte aligned)
        const int32_t stride = (int32_t)((tl->maxMembers + 15) / 16 * 16);
        const size_t smem = (size_t)stride * (sizeof(float4) + sizeof(float2));
#define TILE_LAUNCH(CAPV)                                                                                          \
    k_lj_tile<true, CAPV><<<grid, TILE_ROWS, smem, ctx->stream>>>(                                                \
        rec, tl->members, tl->memberCount, stride, nearList->counts, tl->nearChunks, tl->nearChunksPerRow,  \
        farList->counts, tl->farChunks, tl->farChunksPerRow, rows, nAll, f, tp, ev)
        if (cap)
            TILE_LAUNCH(true);
        else
            TILE_LAUNCH(false);
#undef TILE_LAUNCH
        return after_launch(ctx, "lj_tile");
    }
#define GATHER_LAUNCH(CAPV)                                                                                        \
    k_lj_tile<false, CAPV><<<grid, TILE_ROWS, 0, ctx->stream>>>(                                                  \
        rec, nullptr, nullptr, 0, nearList->counts, nearList->nbrs, nearList->maxNeighbors, farList->counts, \
        farList->nbrs, farList->maxNeighbors, rows, nAll, f, tp, ev)
    if (cap)
        GATHER_LAUNCH(true);
    else
        GATHER_LAUNCH(false);
#undef GATHER_LAUNCH
    return after_launch(ctx, "lj_tile_gather");
}
}  // namespace mrmd_impl
