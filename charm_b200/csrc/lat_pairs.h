// Which latitude pairs of a grid the two-degree recurrence (two.cuh) takes:
// host code of engine.cpp without CUDA in it.
#pragma once

#include <cmath>

namespace cb
{

constexpr double TWO_NEAR = 0.05;      // |sin(lat)| (two.cuh)
// Latitudes of a sphere, with room for the rounding of one in degrees.  A
// grid may hold any angles: beyond this the series of k_geometry do not serve.
constexpr double LAT_MAX = 1.57079632679489661923 + 1e-6;

inline bool latitudes_in_range(const double *lat, int np)
{
    for (int p = 0; p < np; p++)
        if (!(std::fabs(lat[p]) <= LAT_MAX))
            return false;
    return true;
}

// Pairs that the two-degree recurrence may take: |lat| must not grow along
// the pairs (so that neighbouring lanes are neighbouring latitudes and the
// polar form of a 32-pair group fits all of it), from the first pair to the
// first one within TWO_NEAR of the equator.  *polar: the leading pairs, in
// whole groups of 32, poleward of 30 degrees.
inline int two_pairs(const double *lat, int np, int *polar)
{
    const double near = std::asin(TWO_NEAR);
    const double polar_lat = 0.52359877559829887308;   // pi / 6
    int n2 = np;
    for (int p = 0; p < np; p++)
    {
        const double a = std::fabs(lat[p]);
        if (p > 0 && !(a <= std::fabs(lat[p - 1])))
            return 0;
        if (!(a >= near) && n2 == np)
            n2 = p;
    }
    // whole warps: the last up to 31 of them join the others when that leaves
    // the others outside 0.8 TWO_NEAR
    const int whole = (np - n2) / 32 * 32;
    if (n2 < np && whole > 0 && whole < np &&
        std::fabs(lat[np - whole - 1]) >= std::asin(0.8 * TWO_NEAR))
        n2 = np - whole;
    int g = 0;
    while (32 * (g + 1) <= n2 && std::fabs(lat[32 * g + 31]) >= polar_lat)
        g++;
    *polar = 32 * g;
    return n2;
}

} // namespace cb
