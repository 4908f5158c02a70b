// Lennard-Jones internals shared by the pair kernels, LJ_IdealGas and the
// fused stepper.
#pragma once

#include <vector>

#include "common.cuh"

namespace mrmd_impl
{
// Device copy of one type pair's PrecomputedValues plus double-float (hi, lo)
// splits of the factors for the mixed form.
struct LJDev
{
    double ff1, ff2, ef1, ef2;
    double rcSqr, capSqr, capDist, capCoeff, shift, eCap;
    float ff1h, ff1l, ff2h, ff2l;  // ff1 = ff1h + ff1l exactly to ~2^-48
    float ef1f, ef2f, shiftf, rcSqrf;
    float capSqrf, capCoeff_f, eCapf, capDistf;
    float capCoeff_l;  // capCoeff = capCoeff_f + capCoeff_l to ~2^-48
    // low parts of the energy factors (double-float energies of the mixed form)
    float ef1l, ef2l, shiftl, capDistl;
    float eCapShh, eCapShl;  // E(r_cap) - shift
};

inline LJDev to_dev(const mrmd_lj_params& p)
{
    LJDev d{};
    d.ff1 = p.ff1;
    d.ff2 = p.ff2;
    d.ef1 = p.ef1;
    d.ef2 = p.ef2;
    d.rcSqr = p.rcSqr;
    d.capSqr = p.cappingDistanceSqr;
    d.capDist = p.cappingDistance;
    d.capCoeff = p.cappingCoeff;
    d.shift = p.shift;
    d.eCap = p.energyAtCappingPoint;
    d.ff1h = (float)p.ff1;
    d.ff1l = (float)(p.ff1 - (double)d.ff1h);
    d.ff2h = (float)p.ff2;
    d.ff2l = (float)(p.ff2 - (double)d.ff2h);
    d.ef1f = (float)p.ef1;
    d.ef2f = (float)p.ef2;
    d.shiftf = (float)p.shift;
    d.rcSqrf = (float)p.rcSqr;
    d.capSqrf = (float)p.cappingDistanceSqr;
    d.capCoeff_f = (float)p.cappingCoeff;
    d.eCapf = (float)p.energyAtCappingPoint;
    d.capDistf = (float)p.cappingDistance;
    // low parts: each (hi, lo) pair holds the double to ~2^-48
    d.capCoeff_l = (float)(p.cappingCoeff - (double)d.capCoeff_f);
    d.ef1l = (float)(p.ef1 - (double)d.ef1f);
    d.ef2l = (float)(p.ef2 - (double)d.ef2f);
    d.shiftl = (float)(p.shift - (double)d.shiftf);
    d.capDistl = (float)(p.cappingDistance - (double)d.capDistf);
    const double ecs = p.energyAtCappingPoint - p.shift;
    d.eCapShh = (float)ecs;
    d.eCapShl = (float)(ecs - (double)d.eCapShh);
    return d;
}

// computeForceAndEnergy (action/LennardJones.hpp:52-78) in FP64; the
// reciprocal is the correctly rounded one, identical to 1.0 / distSqr.
// The reference's formulae with every rounding explicit (fused
// multiply-adds where a product meets a sum, nothing left to the compiler's
// contraction): the same bits in every kernel that inlines it.
__device__ __forceinline__ void lj_eval_fp64(const LJDev& p, double distSqr, double& ff, double& e)
{
    if (distSqr >= p.capSqr)
    {
        const double frac2 = __drcp_rn(distSqr);
        const double frac6 = __dmul_rn(__dmul_rn(frac2, frac2), frac2);
        ff = __dmul_rn(__dmul_rn(frac6, __fma_rn(p.ff1, frac6, -p.ff2)), frac2);
        e = __fma_rn(frac6, __fma_rn(p.ef1, frac6, -p.ef2), -p.shift);
        return;
    }
    const double dist = __dsqrt_rn(distSqr);
    ff = __ddiv_rn(p.capCoeff, dist);
    e = __dsub_rn(__fma_rn(-__dsub_rn(dist, p.capDist), p.capCoeff, p.eCap), p.shift);
}

// The double's leading bits as a float, truncated to 20 fraction bits: below
// 2^-126 zero, beyond FP32 (and NaN, infinity) NaN.
__device__ __forceinline__ float hi_word_f32(double x)
{
    const uint32_t h = (uint32_t)__double2hiint(x), m = h & 0x7fffffffu;
    uint32_t b = (m - 0x38000000u) << 3;
    b = m < 0x38100000u ? 0u : b;
    b = m >= 0x47f00000u ? 0x7fc00000u : b;
    return __uint_as_float((h & 0x80000000u) | b);
}

// True when the pair is certainly beyond the cutoff: per axis the distance
// of the truncated coordinates less 2^-19 of their magnitudes (the two
// truncations, 2^-20 each, and the FP32 rounding) bounds the true one from
// below.  NaN coordinates are never far.
__device__ __forceinline__ bool surely_beyond(float3 a, const double4& pj, float rcSqrUp)
{
    constexpr float E = 1.9073486328125e-6f;  // 2^-19
    const float bx = hi_word_f32(pj.x), by = hi_word_f32(pj.y), bz = hi_word_f32(pj.z);
    auto least = [](float u, float v) {
        const float d = __fmaf_rn(-E, fabsf(u) + fabsf(v), fabsf(u - v));
        return d < 0.f ? 0.f : d;  // NaN stays NaN
    };
    const float dx = least(a.x, bx), dy = least(a.y, by), dz = least(a.z, bz);
    return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)) > rcSqrUp;
}

// 1/x for x in [2^-340, 2^1000], the correctly rounded one or its neighbour:
// the hardware's approximate reciprocal y and the geometric series of
// 1/(1 - e), e = 1 - x y, up to e^2.  The instruction takes 20 fraction bits of
// x and gives 20 of y: below 2^-20 for what is cut from x and at most 2^-20 for
// the rounding of y, so |e| < 2^-19 (2^-19.9 the largest found).  The rest of
// the series, e^3, is below 2^-57, an eighth of an ulp at most: with the last
// rounding the result is within 0.63 ulp (0.05% of 3.4 million results are not
// the correctly rounded ones).  Three FP64 instructions.
__device__ __forceinline__ double rcp_series(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// Comparisons of doubles on the integer pipe (FP64 comparisons run on the
// FP64 pipe), with the outcome of the FP64 ones for NaN too.
__device__ __forceinline__ bool le_zero(double x)
{
    const long long b = __double_as_longlong(x);
    return b == 0 || (b < 0 && (unsigned long long)b <= 0xfff0000000000000ull);
}

__device__ __forceinline__ bool ge_one(double x)
{
    const long long b = __double_as_longlong(x);
    return b >= 0x3ff0000000000000ll && b <= 0x7ff0000000000000ll;
}

// a > b for a >= 0 or NaN, b >= 0
__device__ __forceinline__ bool gt_nonneg(double a, double b)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(a);
    return u > (unsigned long long)__double_as_longlong(b) && u <= 0x7ff0000000000000ull;
}

// LJ force factor and energy of one pair (the formulae of lj_eval_fp64 with
// the reciprocal of rcp_series, 10 FP64 instructions): the general form
// inside the cap and for r^2 below 2^-340.
__device__ __forceinline__ void lj_eval_series(const LJDev& p, double r2, double& ff, double& e)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(r2);
    if (b < (unsigned long long)__double_as_longlong(p.capSqr) || b < 0x2ab0000000000000ull)
    {
        lj_eval_fp64(p, r2, ff, e);
        return;
    }
    const double u = rcp_series(r2);
    const double u3 = __dmul_rn(__dmul_rn(u, u), u);
    ff = __dmul_rn(__dmul_rn(u3, __fma_rn(p.ff1, u3, -p.ff2)), u);
    e = __fma_rn(u3, __fma_rn(p.ef1, u3, -p.ef2), -p.shift);
}

void lj_force_energy_host(const mrmd_lj_params* t, double distSqr, int64_t typeIdx, double* ff, double* e);
void lj_table_host(mrmd_lj_params* out, int64_t numTypes, const double* cap, const double* rc,
                   const double* sigma, const double* epsilon, int isShifted);

// ------------------------------------------------- double-float helpers --
// Error-free transformations (Knuth TwoSum, Dekker/FMA TwoProd); the pair
// (hi, lo) represents hi + lo with |lo| <= ulp(hi)/2 after renormalisation.
struct df
{
    float h, l;
};

__device__ __forceinline__ df two_sum(float a, float b)
{
    const float s = a + b;
    const float bb = s - a;
    const float e = (a - (s - bb)) + (b - bb);
    return {s, e};
}

__device__ __forceinline__ df fast_two_sum(float a, float b)
{
    const float s = a + b;
    return {s, b - (s - a)};
}

__device__ __forceinline__ df df_mul(df a, df b)
{
    const float p = a.h * b.h;
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ df df_sqr(df a)
{
    const float p = a.h * a.h;
    float e = __fmaf_rn(a.h, a.h, -p);
    e = __fmaf_rn(2.0f * a.h, a.l, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ df df_add(df a, df b)
{
    df s = two_sum(a.h, b.h);
    s.l += a.l + b.l;
    return fast_two_sum(s.h, s.l);
}

// 1/a with one Newton step on the double-float residual.  The seed is the
// hardware's approximate reciprocal (a correctly rounded one would cost a
// multi-instruction sequence and gains nothing: the Newton step squares
// the seed's ~2^-23 error).
__device__ __forceinline__ df df_rcp(df a)
{
    const float y = __fdividef(1.0f, a.h);
    float r = __fmaf_rn(-a.h, y, 1.0f);
    r = __fmaf_rn(-a.l, y, r);
    return fast_two_sum(y, y * r);
}

// sqrt(a) from the approximate reciprocal square root and one Newton
// correction on the exact FMA residual (a > 0)
__device__ __forceinline__ df df_sqrt(df a)
{
    const float q = rsqrtf(a.h);
    const float s = a.h * q;
    const float r = __fmaf_rn(-s, s, a.h) + a.l;
    return fast_two_sum(s, r * (0.5f * q));
}

// compensated accumulator (TwoSum), ~2^-48 relative to the final sum
__device__ __forceinline__ void df_acc(df& s, float x)
{
    const df t = two_sum(s.h, x);
    s.h = t.h;
    s.l += t.l;
}

}  // namespace mrmd_impl

struct mrmd_lj
{
    int64_t numTypes = 1;
    int64_t numTypesIndex = 1;
    double rcSqr = 0.0;
    std::vector<mrmd_lj_params> table;
    mrmd_impl::LJDev p0{};
    mrmd_impl::LJDev* dTable = nullptr;
};

namespace mrmd_impl
{
int lj_apply_fp64(mrmd_ctx* ctx, const mrmd_lj* lj, mrmd_atoms* a, const mrmd_nlist* nl,
                  const mrmd_pred* pred, double* ev, const int32_t* realOf = nullptr);
int lj_apply_mixed(mrmd_ctx* ctx, const mrmd_lj* lj, mrmd_atoms* a, const mrmd_nlist* nl,
                   const mrmd_pred* pred, double* ev);
}  // namespace mrmd_impl
