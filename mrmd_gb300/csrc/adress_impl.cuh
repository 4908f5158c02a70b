// AdResS device helpers shared by LJ_IdealGas, UpdateMolecules and the
// batched replica engine: the Slab weighting function, the region checks and
// the drift-compensation histogram bin.
#pragma once

#include <cmath>
#include <limits>

#include "common.cuh"
#include "lj_impl.cuh"

namespace mrmd_impl
{
constexpr int COMP_BINS = 200;  // LJ_IdealGas.hpp:54

struct SlabDev
{
    double cx;
    double atHalf;  // atomisticRegionHalfDiameter
    double hy;      // hybridRegionDiameter
    double outer;   // atHalf + hy
    double k;       // pi / (2 hy)
    int64_t exponent;
    int32_t abrupt;
};

__device__ __forceinline__ double pow_int(double x, int64_t n)
{
    // util/math.hpp:31-46
    double ww = x, yy = 1.0;
    for (int64_t nn = (n > 0) ? n : -n; nn != 0; nn >>= 1)
    {
        if ((nn & 1) == 1) yy *= ww;
        ww *= ww;
    }
    return (n > 0) ? yy : 1.0 / yy;
}

__device__ __forceinline__ void slab_eval(const SlabDev& s, double x, double& lambda, double& modLambda,
                                          double& gx)
{
    // weighting_function/Slab.hpp:161-187 (+ setSmoothWeightInHY :96-120).
    // Outside the hybrid regions this is one FP64 operation: the comparisons
    // are integer ones on the bits of |dx| (a NaN's lie above infinity's and
    // go on to the weights, like the FP64 comparisons'; to_slab has atHalf and
    // outer such that those with a NaN fail too), and k and outer are the host's,
    // of the same roundings.  The gradient's dx / |dx| is a sign.
    const double dx = x - s.cx;
    const double absDx = fabs(dx);
    const long long b = __double_as_longlong(absDx);
    gx = 0.0;
    if (b < __double_as_longlong(s.atHalf))
    {
        lambda = 1.0;
        modLambda = 1.0;
    }
    else if (b > __double_as_longlong(s.outer) && b <= 0x7ff0000000000000ll)
    {
        lambda = 0.0;
        modLambda = 0.0;
    }
    else if (s.abrupt)
    {
        lambda = 1.0;
        modLambda = 1.0;
    }
    else
    {
        double sn, base;
        sincos(s.k * (absDx - s.atHalf), &sn, &base);
        lambda = base * base;
        modLambda = pow_int(base, s.exponent);
        const double slope = s.k * (double)s.exponent * sn * pow_int(base, s.exponent - 1);
        gx = __double_as_longlong(dx) < 0 ? slope : -slope;
    }
}

// CheckRegion.hpp:25-38 with REGION_CHECK_EPSILON = 0
__device__ __forceinline__ bool is_at(double l) { return ge_one(l); }
__device__ __forceinline__ bool is_cg(double l) { return le_zero(l); }
__device__ __forceinline__ bool is_hy(double l) { return !is_at(l) && !is_cg(l); }

__device__ __forceinline__ int comp_bin(double lambda)
{
    // MultiHistogram(0, 1, 200).getBin (data/MultiHistogram.hpp:60-66)
    const double inv = 1.0 / ((1.0 - 0.0) / (double)COMP_BINS);
    int64_t b = __double2ll_rd(lambda * inv);
    if (b < 0 || b >= COMP_BINS) return -1;
    return (int)b;
}

inline SlabDev to_slab(const mrmd_slab* s)
{
    // Slab constructor, weighting_function/Slab.hpp:189-200
    SlabDev d{};
    d.cx = s->center[0];
    d.atHalf = 0.5 * s->atomisticRegionDiameter;
    d.hy = s->hybridRegionDiameter;
    d.outer = d.atHalf + d.hy;
    d.k = 3.141592653589793238462643383279502884 / (2.0 * d.hy);
    // a NaN diameter: no |dx| lies below atHalf or above outer, and the weights
    // are NaN (slab_eval compares bits: a positive NaN's lie above all others)
    if (std::isnan(d.outer)) d.outer = std::numeric_limits<double>::quiet_NaN();
    if (std::isnan(d.atHalf))
    {
        d.atHalf = -1.0;
        d.k = std::numeric_limits<double>::quiet_NaN();
    }
    d.exponent = 2 * s->nu;
    d.abrupt = s->interfaceType == 1;
    return d;
}
}  // namespace mrmd_impl
