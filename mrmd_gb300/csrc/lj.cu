// action::LennardJones: capped, optionally shifted LJ on a half Verlet list.
//
// FP64 form: the j-force is scattered with FP64 atomics into the 32-byte atom
// sector (atoms are cell-sorted by the stepper, so a warp's neighbours share
// cache lines), energy and virial are reduced per block and added once per
// block.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "lj_impl.cuh"
#include "nlist_impl.cuh"

using namespace mrmd_impl;

namespace mrmd_impl
{
void lj_force_energy_host(const mrmd_lj_params* t, double distSqr, int64_t typeIdx, double* ff, double* e)
{
    // action/LennardJones.hpp:52-78 evaluated on the host with IEEE doubles
    const mrmd_lj_params& p = t[typeIdx];
    if (distSqr >= p.cappingDistanceSqr)
    {
        const double frac2 = 1.0 / distSqr;
        const double frac6 = frac2 * frac2 * frac2;
        *ff = frac6 * (p.ff1 * frac6 - p.ff2) * frac2;
        *e = frac6 * (p.ef1 * frac6 - p.ef2) - p.shift;
        return;
    }
    const double dist = std::sqrt(distSqr);
    *ff = p.cappingCoeff / dist;
    *e = p.energyAtCappingPoint - (dist - p.cappingDistance) * p.cappingCoeff - p.shift;
}

void lj_table_host(mrmd_lj_params* out, int64_t numTypes, const double* cap, const double* rc,
                   const double* sigma, const double* epsilon, int isShifted)
{
    // constructor action/LennardJones.cpp:81-116, precompute :61-79
    for (int64_t t = 0; t < numTypes * numTypes; ++t)
    {
        const double sig2 = sigma[t] * sigma[t];
        const double sig6 = sig2 * sig2 * sig2;
        std::memset(&out[t], 0, sizeof(mrmd_lj_params));
        out[t].ff1 = 48.0 * epsilon[t] * sig6 * sig6;
        out[t].ff2 = 24.0 * epsilon[t] * sig6;
        out[t].ef1 = 4.0 * epsilon[t] * sig6 * sig6;
        out[t].ef2 = 4.0 * epsilon[t] * sig6;
        out[t].rcSqr = rc[t] * rc[t];
        out[t].cappingDistance = cap[t];
    }
    for (int64_t t = 0; t < numTypes * numTypes; ++t)
    {
        const double capDist = out[t].cappingDistance;
        out[t].cappingDistance = 0.0;
        out[t].cappingDistanceSqr = 0.0;
        double ff, e;
        lj_force_energy_host(out, capDist * capDist, t, &ff, &e);
        out[t].cappingCoeff = ff * capDist;
        out[t].energyAtCappingPoint = e;
        out[t].cappingDistance = capDist;
        out[t].cappingDistanceSqr = capDist * capDist;
        if (isShifted)
        {
            lj_force_energy_host(out, out[t].rcSqr, t, &ff, &e);
            out[t].shift = e;
        }
    }
}

namespace
{
constexpr int LJ_TB = 128;
constexpr int LJ_CHUNK = 64;  // list entries of a row scanned at a time
constexpr int LJ_BLOCKS = 5;  // resident blocks per SM: with 6 or 7 the segments take the L1's room
                              // (4,000,000 atoms: 4.83 ms with 5, 4.89 with 6, 5.03 with 7)

// Pair force on the half list in two phases per warp, R list rows per warp.
//
// The kernel is bound by the FP64 pipe (2 lanes per SM and clock on GB300),
// so it is laid out to issue as few FP64 instructions as possible, with all
// 32 lanes busy in each:
//  1. Scan: the rows' entries are tested against the cutoff in FP32 from the
//     high words of the coordinates (a lower bound of r^2, surely_beyond);
//     the ones that may be in range (71% with a skin of 0.3 at 2.5) are
//     appended to their row's segment in shared memory.
//  2. Evaluation: the segments' pairs, numbered row after row, are dealt out
//     evenly, so that every lane evaluates the same number of pairs (+-1)
//     whatever the rows' lengths; a lane keeps the force of its current row
//     in registers and adds it to the row's atom when it moves on.
// A pair takes 22 FP64 instructions: distance 3, r^2 3, reciprocal 3, force
// factor 5, energy and virial sums 2 (of u^3 and u^6; E and W are formed once
// per lane), forces 6.  The comparisons are integer ones on the bits.
// One lane per row with all entries in FP64 and a correctly rounded
// reciprocal took ~35 instructions per entry and, with rows of unequal
// length, 47 rounds for 38 entries.  At 256,000 atoms 4.91e6 FP64 warp
// instructions (22 per pair in range are 4.85e6), FP64 pipe 76% active.
// Measured times: lj_rows_per_warp.
//
// realOf (may be null): the real atom of every ghost; a ghost's force then goes
// straight to it, and no fold-back follows (its pass over all atoms, bound by
// its dependent loads, took 9 us of a 4,000-atom step and 20 at 256,000).
template <bool PRED, bool MULTI, int R>
__global__ void __launch_bounds__(LJ_TB, LJ_BLOCKS) k_lj_fp64(
    const double4* __restrict__ pos, double* __restrict__ force, const int32_t* __restrict__ type,
    const LJDev p0, const LJDev* __restrict__ table, int32_t numTypesIndex, double rcSqr, float rcSqrUp,
    const int32_t* __restrict__ counts, const int32_t* __restrict__ nbrs, int64_t cap, int64_t n,
    int64_t begin, int64_t nAll, mrmd_dev::Pred pred, const int32_t* __restrict__ realOf, int64_t nLocal,
    double* __restrict__ ev)
{
    constexpr int G = 32 / R;  // lanes scanning one row
    constexpr unsigned ALL = 0xffffffffu;
    constexpr unsigned ROW0 = R == 2 ? 0x55555555u : R == 4 ? 0x11111111u : R == 8 ? 0x01010101u : 0x00010001u;  // row 0's lanes
    static_assert(R == 2 || R == 4 || R == 8 || R == 16, "rows per warp");
    __shared__ int32_t segS[LJ_TB / 32][LJ_CHUNK * R];
    __shared__ int32_t endS[LJ_TB / 32][R];
    __shared__ double red[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t* seg = segS[warp];  // entry q of row r: seg[q * R + r]
    int32_t* ends = endS[warp];
    // sums over the lane's pairs: u^3, u^6 and the number of uncapped pairs;
    // energies and force factor * r^2 of the others
    double s3 = 0.0, s6 = 0.0, sE = 0.0, sW = 0.0;
    int32_t num = 0;
    const unsigned long long rcBits = (unsigned long long)__double_as_longlong(rcSqr);
    const int r = lane % R, g = lane / R;
    // a warp takes every (number of warps)-th group of R rows
    for (int64_t row0 = (blockIdx.x * (int64_t)(LJ_TB / 32) + warp) * R; row0 < n;
         row0 += (int64_t)gridDim.x * (LJ_TB / 32) * R)
    {
        const int64_t row = row0 + r;
        const int32_t cnt = row < n ? counts[row] : 0;
        int32_t maxCnt = cnt;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) maxCnt = max(maxCnt, __shfl_xor_sync(ALL, maxCnt, o));
        double4 pr = make_double4(0.0, 0.0, 0.0, 0.0);
        if (cnt > 0) pr = pos[begin + row];
        const float3 pf = make_float3(hi_word_f32(pr.x), hi_word_f32(pr.y), hi_word_f32(pr.z));
        const int32_t* __restrict__ col = nbrs + mrmd_dev::nbr_row(row, cap);
        for (int32_t k0 = 0; k0 < maxCnt; k0 += LJ_CHUNK)
        {
            // 1. scan
            int32_t c = 0;  // entries of the row kept so far (the same in its G lanes)
            const int32_t kEnd = min(k0 + LJ_CHUNK, maxCnt);
#pragma unroll 4
            for (int32_t kk = k0; kk < kEnd; kk += G)
            {
                const int32_t k = kk + g;
                bool keep = k < cnt;
                int32_t j = 0;
                if (keep)
                {
                    j = __ldg(col + 32 * (int64_t)k);
                    keep = MRMD_IN_BOUNDS(j, nAll);
                    if (keep)
                    {
                        const double4 pj = mrmd_dev::ldg4(pos + j);
                        keep = !surely_beyond(pf, pj, rcSqrUp);
                        if (PRED) keep = keep && mrmd_dev::pred2(pred, pr.x, pr.y, pr.z, pj.x, pj.y, pj.z);
                    }
                }
                const unsigned m = __ballot_sync(ALL, keep) & (ROW0 << r);
                if (keep) seg[(c + __popc(m & ((1u << lane) - 1u))) * R + r] = j;
                c += __popc(m);
            }
            // 2. evaluation: row r's pairs are numbers [incl - c, incl)
            int32_t incl = c;
#pragma unroll
            for (int o = 1; o < R; o <<= 1)
            {
                const int32_t t = __shfl_up_sync(ALL, incl, o, R);
                if (r >= o) incl += t;
            }
            if (g == 0) ends[r] = incl;
            __syncwarp();
            const int32_t total = ends[R - 1];
            int32_t t = (total * lane) >> 5;  // total <= R * LJ_CHUNK
            const int32_t tEnd = (total * (lane + 1)) >> 5;
            if (t < tEnd)
            {
                int32_t q = 0, qStart = 0, qEnd;  // current row and its numbers
                {
                    int lo = 0, hi = R - 1;  // first row that ends above t
                    while (lo < hi)
                    {
                        const int mid = (lo + hi) >> 1;
                        if (ends[mid] > t) hi = mid;
                        else lo = mid + 1;
                    }
                    q = lo;
                    qStart = q > 0 ? ends[q - 1] : 0;
                    qEnd = ends[q];
                }
                int64_t i = begin + row0 + q;
                double4 pi = mrmd_dev::ldg4(pos + i);
                int32_t ti = MULTI ? type[i] * numTypesIndex : 0;
                double fx = 0.0, fy = 0.0, fz = 0.0;
                for (; t < tEnd; ++t)
                {
                    if (t >= qEnd)
                    {
                        atomicAdd(force + 4 * i + 0, fx);
                        atomicAdd(force + 4 * i + 1, fy);
                        atomicAdd(force + 4 * i + 2, fz);
                        fx = fy = fz = 0.0;
                        do
                        {
                            ++q;
                            qStart = qEnd;
                            qEnd = ends[q];
                        } while (t >= qEnd);
                        i = begin + row0 + q;
                        pi = mrmd_dev::ldg4(pos + i);
                        if (MULTI) ti = type[i] * numTypesIndex;
                    }
                    const int64_t j = seg[(t - qStart) * R + q];
                    const double4 pj = mrmd_dev::ldg4(pos + j);
                    const double dx = pi.x - pj.x;
                    const double dy = pi.y - pj.y;
                    const double dz = pi.z - pj.z;
                    const double r2 = __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
                    // bits of a non-negative double order as the value; a NaN's
                    // lie above infinity's and are not skipped
                    const unsigned long long b = (unsigned long long)__double_as_longlong(r2);
                    if (b > rcBits && b <= 0x7ff0000000000000ull) continue;
                    const LJDev& p = MULTI ? table[ti + type[j]] : p0;
                    double ff;
                    if (b >= (unsigned long long)__double_as_longlong(p.capSqr) && b >= 0x2ab0000000000000ull)  // 2^-340
                    {
                        const double u = rcp_series(r2);
                        const double u3 = __dmul_rn(__dmul_rn(u, u), u);
                        ff = __dmul_rn(__dmul_rn(u3, __fma_rn(p.ff1, u3, -p.ff2)), u);
                        if (MULTI)
                        {
                            sE += __fma_rn(u3, __fma_rn(p.ef1, u3, -p.ef2), -p.shift);
                            sW = __fma_rn(ff, r2, sW);
                        }
                        else
                        {
                            s3 += u3;
                            s6 = __fma_rn(u3, u3, s6);
                            ++num;
                        }
                    }
                    else
                    {
                        double e;
                        lj_eval_fp64(p, r2, ff, e);
                        sE += e;
                        sW = __fma_rn(ff, r2, sW);
                    }
                    const double gx = __dmul_rn(dx, -ff), gy = __dmul_rn(dy, -ff), gz = __dmul_rn(dz, -ff);
                    fx -= gx;
                    fy -= gy;
                    fz -= gz;
                    const int64_t to = realOf && j >= nLocal ? (int64_t)realOf[j] : j;
                    if (!MRMD_IN_BOUNDS(to, realOf ? nLocal : nAll)) continue;
                    double* fj = force + 4 * to;
                    atomicAdd(fj + 0, gx);
                    atomicAdd(fj + 1, gy);
                    atomicAdd(fj + 2, gz);
                }
                atomicAdd(force + 4 * i + 0, fx);
                atomicAdd(force + 4 * i + 1, fy);
                atomicAdd(force + 4 * i + 2, fz);
            }
            __syncwarp();  // the next chunk overwrites the segments
        }
    }
    if (!MULTI)
    {
        // E = sum ef1 u^6 - ef2 u^3 - shift, -2 W = sum ff1 u^6 - ff2 u^3
        // (action/LennardJones.hpp:52-78: forceFactor r^2 = ff1 u^6 - ff2 u^3)
        sE += __fma_rn(p0.ef1, s6, -__fma_rn(p0.ef2, s3, __dmul_rn(p0.shift, (double)num)));
        sW += __fma_rn(p0.ff1, s6, -__dmul_rn(p0.ff2, s3));
    }
    mrmd_dev::block_sum2(sE, sW, red);
    if (threadIdx.x == 0)
    {
        atomicAdd(ev + 0, sE);
        atomicAdd(ev + 1, -0.5 * sW);
    }
}

// Rows per warp.  Few rows give a small system enough warps; many rows make
// the evaluation's rounds full (27.6 pairs in range per row at density
// 0.8442 against 32 lanes) and amortise the force additions at row changes.
// Kernel times in us for 2 / 4 / 8 / 16 rows (one lane per row, all entries
// in FP64, before), dense fluid:
//       2,048 atoms   10.6 / 12.6 / 18.8 / 29.1   (76)
//       4,000         16.6 / 14.6 / 18.6 / 29.0   (76)
//      10,976         28.9 / 26.9 / 29.0 / 39.0
//      32,000         59.6 / 57.5 / 55.6 / 63.7   (120)
//     256,000          377 /  363 /  330 /  330   (782)
//   4,000,000         5640 / 5430 / 4930 / 4830   (11332)
// (1 row: 12.7 us at 2,048; 32 rows: 4900 us at 4,000,000).  The FP64
// instructions of the pairs alone take 3.86 ms at 4,000,000 atoms.
int lj_rows_per_warp(const mrmd_ctx* ctx, int64_t n)
{
    const int64_t sms = ctx->numSMs;
    if (n >= 16 * 96 * sms) return 16;  // 96 warps per SM and more
    if (n >= 8 * 16 * sms) return 8;
    if (n >= 4 * 5 * sms) return 4;
    return 2;
}
}  // namespace

int lj_apply_fp64(mrmd_ctx* ctx, const mrmd_lj* lj, mrmd_atoms* a, const mrmd_nlist* nl,
                  const mrmd_pred* pred, double* ev, const int32_t* realOf)
{
    const int64_t n = nl->rows;
    if (n == 0) return MRMD_OK;
    const bool usePred = pred != nullptr && pred->kind != MRMD_PRED_ALWAYS;
    const bool multi = lj->numTypes > 1;
    const mrmd_dev::Pred dp = to_dev_pred(pred);
    const double4* pos = reinterpret_cast<const double4*>(a->pos);
    const float rcSqrUp = (float)(lj->rcSqr * (1.0 + 1e-6));
    auto launch = [&](auto kernel, int R) {
        const int64_t groups = div_up(n, (int64_t)(LJ_TB / 32) * R), most = (int64_t)ctx->numSMs * LJ_BLOCKS;
        const unsigned grid = (unsigned)(groups < most ? groups : most);
        kernel<<<grid, LJ_TB, 0, ctx->stream>>>(pos, a->force, a->type, lj->p0, lj->dTable, (int32_t)lj->numTypesIndex,
                                                lj->rcSqr, rcSqrUp, nl->counts, nl->nbrs, nl->maxNeighbors, n,
                                                nl->begin, a->numLocal + a->numGhost, dp, realOf, a->numLocal, ev);
    };
#define LJ_ROWS(R)                                              \
    if (usePred && multi) launch(k_lj_fp64<true, true, R>, R);  \
    else if (usePred) launch(k_lj_fp64<true, false, R>, R);     \
    else if (multi) launch(k_lj_fp64<false, true, R>, R);       \
    else launch(k_lj_fp64<false, false, R>, R)
    switch (lj_rows_per_warp(ctx, n))
    {
        case 16: LJ_ROWS(16); break;
        case 8: LJ_ROWS(8); break;
        case 4: LJ_ROWS(4); break;
        default: LJ_ROWS(2); break;
    }
#undef LJ_ROWS
    return after_launch(ctx, "lj_fp64");
}
}  // namespace mrmd_impl

extern "C" {

int mrmd_lj_create(mrmd_ctx* ctx, mrmd_lj** out, int64_t numTypes, int64_t numTypesIndex,
                   const double* cappingDistance, const double* rc, const double* sigma,
                   const double* epsilon, int isShifted)
{
    if (!ctx || !out || !cappingDistance || !rc || !sigma || !epsilon) return MRMD_ERR_ARG;
    MRMD_CHECK_ARG(numTypes >= 1 && numTypes <= 64, ctx, "numTypes out of range");
    MRMD_CHECK_ARG(numTypesIndex >= 0 && numTypesIndex <= numTypes, ctx, "bad numTypesIndex");
    *out = nullptr;
    mrmd_lj* lj = new mrmd_lj();
    lj->numTypes = numTypes;
    lj->numTypesIndex = numTypesIndex;
    const int64_t n2 = numTypes * numTypes;
    lj->table.resize((size_t)n2);
    lj_table_host(lj->table.data(), numTypes, cappingDistance, rc, sigma, epsilon, isShifted);
    double rcMax = rc[0];
    for (int64_t t = 1; t < n2; ++t) rcMax = std::fmax(rcMax, rc[t]);
    lj->rcSqr = rcMax * rcMax;  // action/LennardJones.cpp:54-55
    std::vector<LJDev> dev((size_t)n2);
    for (int64_t t = 0; t < n2; ++t) dev[(size_t)t] = to_dev(lj->table[(size_t)t]);
    lj->p0 = dev[0];
    int rc2 = dmalloc(ctx, reinterpret_cast<void**>(&lj->dTable), sizeof(LJDev) * (size_t)n2);
    if (rc2 == MRMD_OK)
        rc2 = h2d(ctx, lj->dTable, dev.data(), sizeof(LJDev) * (size_t)n2);
    if (rc2 != MRMD_OK)
    {
        dfree(lj->dTable);
        delete lj;
        return rc2;
    }
    *out = lj;
    return MRMD_OK;
}

int mrmd_lj_destroy(mrmd_ctx* ctx, mrmd_lj* lj)
{
    if (!lj) return MRMD_OK;
    if (ctx) cudaStreamSynchronize(ctx->stream);
    dfree(lj->dTable);
    delete lj;
    return MRMD_OK;
}

int mrmd_lj_get_params(const mrmd_lj* lj, mrmd_lj_params* out, int64_t count)
{
    if (!lj || !out) return MRMD_ERR_ARG;
    const int64_t n = (int64_t)lj->table.size();
    for (int64_t t = 0; t < count && t < n; ++t) out[t] = lj->table[(size_t)t];
    return MRMD_OK;
}

int mrmd_lj_apply(mrmd_ctx* ctx, mrmd_lj* lj, mrmd_atoms* a, const mrmd_nlist* nl, const mrmd_pred* pred,
                  int precision, double* energy, double* virial)
{
    if (!ctx || !lj || !a || !nl) return MRMD_ERR_ARG;
    MRMD_CHECK_ARG(pred_valid(pred), ctx, "bad predicate");
    MRMD_CHECK_ARG(precision == MRMD_PREC_FP64 || precision == MRMD_PREC_MIXED, ctx, "bad precision");
    MRMD_TRY(check_list_fits(ctx, nl, a->numLocal, a->numLocal + a->numGhost));
    double* ev = ctx->devScalars + 16;
    MRMD_CUDA(ctx, cudaMemsetAsync(ev, 0, 2 * sizeof(double), ctx->stream));
    if (precision == MRMD_PREC_FP64)
        MRMD_TRY(lj_apply_fp64(ctx, lj, a, nl, pred, ev));
    else
        MRMD_TRY(lj_apply_mixed(ctx, lj, a, nl, pred, ev));
    if (energy || virial)
    {
        MRMD_CUDA(ctx, cudaMemcpyAsync(ctx->hostScalars + 16, ev, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                                       ctx->stream));
        MRMD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (energy) *energy = ctx->hostScalars[16];
        if (virial) *virial = ctx->hostScalars[17];
        return MRMD_OK;
    }
    return finish(ctx, "lj_apply");
}

}  // extern "C"
