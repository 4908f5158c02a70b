// Mixed-precision Lennard-Jones pair force.
//
// Positions stay FP64 in the atoms; before the pair kernel each coordinate
// c = x - origin (origin = the list's cell-grid corner) is split into
//   hi = c rounded to a multiple of 2^-q, q = 24 - ceil(log2(extent)),
//   lo = float(c - hi),
// so every hi is an integer multiple of 2^-q below 2^24 * 2^-q: the FP32
// difference hi_i - hi_j is exact, and dx = (hi_i - hi_j) + (lo_i - lo_j)
// carries ~2^-40 absolute accuracy.  r^2, 1/r^2, the force factor and the
// force products are evaluated in double-float (pairs of FP32), because the
// LJ force factor amplifies a relative error of r^2 sevenfold (F ~ r^-14) and
// single pair forces can exceed the atom's net force by orders of magnitude;
// the per-atom sums are compensated double-float.  All of this runs on the
// FP32 pipe.  Energy and virial use FP32 terms, summed with compensated FP32
// per thread and FP64 across threads.
#include <cmath>

#include "common.cuh"
#include "lj_impl.cuh"
#include "lj_mixed.cuh"
#include "nlist_impl.cuh"

using namespace mrmd_impl;

namespace mrmd_impl
{
SplitParams split_params(const double* origin, double extent)
{
    SplitParams s{};
    int e = 0;
    std::frexp(extent > 1.0 ? extent : 1.0, &e);  // extent < 2^e
    const int q = 24 - e;
    s = make_split(std::ldexp(1.0, q), std::ldexp(1.0, -q));
    s.origin = make_double3(origin[0], origin[1], origin[2]);
    return s;
}

__global__ void k_split_coords(const double4* __restrict__ pos, int64_t n, SplitParams sp,
                               float4* __restrict__ hi, float4* __restrict__ lo, int stride)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        const double4 p = pos[i];
        float4 h, l;
        split_one(p.x - sp.origin.x, sp, h.x, l.x);
        split_one(p.y - sp.origin.y, sp, h.y, l.y);
        split_one(p.z - sp.origin.z, sp, h.z, l.z);
        h.w = 0.0f;
        l.w = 0.0f;
        hi[i * stride] = h;
        lo[i * stride] = l;
    }
}

int split_coords(mrmd_ctx* ctx, const double* pos4, int64_t n, const SplitParams& sp, float4* hi, float4* lo,
                 int stride)
{
    if (n == 0) return MRMD_OK;
    k_split_coords<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(reinterpret_cast<const double4*>(pos4), n, sp,
                                                                   hi, lo, stride);
    return after_launch(ctx, "split_coords");
}

namespace
{
constexpr int MX_TB = 128;

struct Acc
{
    df fx{0.f, 0.f}, fy{0.f, 0.f}, fz{0.f, 0.f}, e{0.f, 0.f}, w{0.f, 0.f};

    __device__ __forceinline__ void add(const PairMixed& q)
    {
        df_acc_prod(fx, q.dh.x, q.dl.x, q.ff);
        df_acc_prod(fy, q.dh.y, q.dl.y, q.ff);
        df_acc_prod(fz, q.dh.z, q.dl.z, q.ff);
        df_acc(e, q.e);
        df_acc(w, -0.5f * q.ff.h * q.r2h);
    }

};

constexpr int MX_CHUNK = 40;  // list entries of a row scanned at a time

// One list row per LANES lanes.  As in the FP64 kernel the row's entries are
// tested first (on the heads of the split coordinates, which bound r from
// below: each component's low parts differ by at most one quantum), then the
// ones that may be in range are dealt to the row's lanes; the evaluation is
// some 200 FP32 instructions, and a third of the entries are out of range.
// The forces become doubles by integer conversions (two FP64 conversions and
// an addition per component before: the FP64 pipe bound the kernel).
// Measured times: lj_mixed_half.
template <bool PRED, int LANES>
__global__ void __launch_bounds__(MX_TB) k_lj_mixed_half(
    const float4* __restrict__ hi, const float4* __restrict__ lo, const double4* __restrict__ pos,
    double* __restrict__ force, const LJDev p, RcSq rc2, float rcReach, const int32_t* __restrict__ counts,
    const int32_t* __restrict__ nbrs, int64_t cap, int64_t n, int64_t begin, int64_t nAll, mrmd_dev::Pred pred,
    double* __restrict__ ev)
{
    constexpr unsigned ALL = 0xffffffffu;
    __shared__ double red[64];
    __shared__ uint8_t segS[MX_TB / LANES][MX_CHUNK];
    const int lane = threadIdx.x & 31, sub = lane % LANES;
    const unsigned mine = (LANES == 32 ? ALL : ((1u << LANES) - 1u)) << (lane & ~(LANES - 1));
    const unsigned before = mine & ((1u << lane) - 1u);
    uint8_t* seg = segS[threadIdx.x / LANES];
    Acc acc;
    const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
    const bool live = row < n;
    // list row `row` belongs to particle begin + row (the list's range)
    const int64_t i = begin + (live ? row : 0);
    const float4 hi_i = hi[i], lo_i = lo[i];
    double4 pi;
    if (PRED) pi = pos[i];
    const int32_t cnt = live ? counts[row] : 0;
    const int32_t* __restrict__ col = nbrs + mrmd_dev::nbr_row(live ? row : 0, cap);
    int32_t most = cnt;
#pragma unroll
    for (int o = 16; o >= LANES; o >>= 1) most = max(most, __shfl_xor_sync(ALL, most, o));
    for (int32_t k0 = 0; k0 < most; k0 += MX_CHUNK)
    {
        int32_t kept = 0;
        const int32_t kEnd = min(k0 + MX_CHUNK, most);
#pragma unroll 4
        for (int32_t kk = k0; kk < kEnd; kk += LANES)
        {
            const int32_t k = kk + sub;
            bool keep = k < cnt;
            if (keep)
            {
                const int32_t j = __ldg(col + 32 * (int64_t)k);
                keep = MRMD_IN_BOUNDS(j, nAll);
                if (keep)
                {
                    const float4 hj = __ldg(hi + j);
                    const float dx = hi_i.x - hj.x, dy = hi_i.y - hj.y, dz = hi_i.z - hj.z;
                    keep = !(__fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)) > rcReach);
                    if (PRED && keep)
                    {
                        const double4 pj = mrmd_dev::ldg4(pos + j);
                        keep = mrmd_dev::pred2(pred, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z);
                    }
                }
            }
            const unsigned m = __ballot_sync(ALL, keep);
            if (keep) seg[kept + __popc(m & before)] = (uint8_t)(k - k0);
            kept += __popc(m & mine);
        }
        __syncwarp();
        for (int32_t q = sub; q < kept; q += LANES)
        {
            const int32_t j = __ldg(col + 32 * (int64_t)(k0 + seg[q]));
            PairMixed f;
            if (!pair_mixed(hi_i, lo_i, __ldg(hi + j), __ldg(lo + j), p, rc2, f)) continue;
            acc.add(f);
            // -(dh + dl) ff: the product of the turned force factor
            const df nff = {-f.ff.h, -f.ff.l};
            atomicAdd(force + 4 * (int64_t)j + 0, prod_d(f.dh.x, f.dl.x, nff));
            atomicAdd(force + 4 * (int64_t)j + 1, prod_d(f.dh.y, f.dl.y, nff));
            atomicAdd(force + 4 * (int64_t)j + 2, prod_d(f.dh.z, f.dl.z, nff));
        }
        __syncwarp();
    }
    double g[3] = {__dadd_rn(f32_to_f64(acc.fx.h), f32_to_f64(acc.fx.l)),
                   __dadd_rn(f32_to_f64(acc.fy.h), f32_to_f64(acc.fy.l)),
                   __dadd_rn(f32_to_f64(acc.fz.h), f32_to_f64(acc.fz.l))};
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1)
#pragma unroll
        for (int d = 0; d < 3; ++d) g[d] += __shfl_xor_sync(ALL, g[d], o);
    if (live && sub == 0)
#pragma unroll
        for (int d = 0; d < 3; ++d) atomicAdd(force + 4 * i + d, g[d]);
    double e = __dadd_rn(f32_to_f64(acc.e.h), f32_to_f64(acc.e.l));
    double w = __dadd_rn(f32_to_f64(acc.w.h), f32_to_f64(acc.w.l));
    mrmd_dev::block_sum2(e, w, red);
    if (threadIdx.x == 0)
    {
        atomicAdd(ev + 0, e);
        atomicAdd(ev + 1, w);
    }
}

}  // namespace

int lj_mixed_half(mrmd_ctx* ctx, const float4* hi, const float4* lo, const mrmd_lj* lj, mrmd_atoms* a,
                  const mrmd_nlist* nl, const mrmd_pred* pred, double* ev)
{
    const int64_t n = nl->rows;
    if (n == 0) return MRMD_OK;
    const bool usePred = pred != nullptr && pred->kind != MRMD_PRED_ALWAYS;
    const mrmd_dev::Pred dp = to_dev_pred(pred);
    const RcSq rc2 = make_rcsq(lj->rcSqr);
    const double4* pos = reinterpret_cast<const double4*>(a->pos);
    // |dl| is at most one quantum per component: a pair within rc has heads
    // within rc + sqrt(3) quanta
    const double reach = std::sqrt(lj->rcSqr) + 1.7320509 * split_params_for(nl).invScale;
    const float rcReach = (float)(reach * reach * (1.0 + 1e-6));
    auto launch = [&](auto kernel, int lanes) {
        kernel<<<(unsigned)div_up(n * lanes, MX_TB), MX_TB, 0, ctx->stream>>>(
            hi, lo, pos, a->force, lj->p0, rc2, rcReach, nl->counts, nl->nbrs, nl->maxNeighbors, n, nl->begin,
            a->numLocal + a->numGhost, dp, ev);
    };
#define MX_LANES(L)                                       \
    if (usePred) launch(k_lj_mixed_half<true, L>, L);     \
    else launch(k_lj_mixed_half<false, L>, L)
    // lanes per row: us with 1 / 2 / 4 / 8 lanes (one lane per row, every entry
    // evaluated, FP64 conversions, before)
    //       4,000 atoms   50 /  31 /  23 /  19   (60)
    //      32,000         53 /  40 /  37 /  44   (69)
    //      87,808         80 /  73 /  71 /  83   (125)
    //     256,000        185 / 158 / 161 / 204   (327)
    //   4,000,000       2112 / 2030 / 2235 / 2958   (4536)
    // With rows of a few entries (a gas) a second lane of a large system has
    // nothing to do: us of the call with 1 / 2 lanes at random placement, 256,000
    // atoms and 0.2 / 0.9 / 2.3 / 4.6 / 9.2 entries a row 44 / 54, 52 / 66, 66 /
    // 66, 78 / 79, 103 / 102, 1,000,000 atoms 106 / 151, 127 / 176, 152 / 192,
    // 191 / 217, 274 / 287 (139, 178, 238, 315, 460 before)
    const int64_t sms = ctx->numSMs;
    if (n < 40 * sms)
    {
        MX_LANES(8);
    }
    else if (n < 640 * sms)
    {
        MX_LANES(4);
    }
    else if (nl->totalPairs >= 4 * n)
    {
        MX_LANES(2);
    }
    else
    {
        MX_LANES(1);
    }
#undef MX_LANES
    return after_launch(ctx, "lj_mixed_half");
}

SplitParams split_params_for(const mrmd_nlist* nl)
{
    const CellList* cl = static_cast<const CellList*>(nl->cells);
    const double origin[3] = {cl->g.mn.x, cl->g.mn.y, cl->g.mn.z};
    return split_params(origin, cl->g.extent * 1.25 + 8.0);
}

int lj_apply_mixed(mrmd_ctx* ctx, const mrmd_lj* lj, mrmd_atoms* a, const mrmd_nlist* nl, const mrmd_pred* pred,
                   double* ev)
{
    if (lj->numTypes > 1) return set_error(ctx, MRMD_ERR_ARG, "mixed precision supports one atom type");
    if (nl->rows == 0) return MRMD_OK;
    const SplitParams sp = split_params_for(nl);
    const int64_t nAll = a->numLocal + a->numGhost;
    float4* hi = static_cast<float4*>(scratch(ctx, sizeof(float4) * 2 * (size_t)nAll));
    if (!hi) return MRMD_ERR_OOM;
    float4* lo = hi + nAll;
    MRMD_TRY(split_coords(ctx, a->pos, nAll, sp, hi, lo));
    return lj_mixed_half(ctx, hi, lo, lj, a, nl, pred, ev);
}
}  // namespace mrmd_impl
