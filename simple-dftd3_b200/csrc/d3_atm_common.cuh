// Smooth cutoff and triple ownership of the three-body kernels (d3_atm.cu) and
// of the pairwise decomposition (d3_pairwise.cu), and the fixed-point sums of the
// former (read by d3_molecule.cu as well).
#pragma once

#include <cfloat>

#include "d3_device.cuh"

namespace d3 {
namespace {

template <class R>
__device__ __forceinline__ void smooth(R r, R cutoff, R width, R& sw, R& dsw)
{
    // cutoff.f90:73-99
    if (width <= R(0) || width >= cutoff) { sw = R(1); dsw = R(0); return; }
    const R inner = cutoff - width;
    if (r <= inner) { sw = R(1); dsw = R(0); }
    else if (r >= cutoff) { sw = R(0); dsw = R(0); }
    else {
        const R x = (cutoff - r) / width;
        sw = x * x * x * (R(10) + x * (R(-15) + R(6) * x));
        dsw = R(-30) * x * x * (R(1) - x) * (R(1) - x) / width;
    }
}

__device__ __forceinline__ bool owns_pair_atm(const Partition& p, int i, int j)
{
    long long hi = i > j ? i : j, lo = i > j ? j : i;
    return (hi * (hi + 1) / 2 + lo) % p.nparts == p.part;
}

// Deterministic accumulation of sums from many warps: a value is added as two
// 64-bit integers, its nearest multiple of 2^-40 and the rest rounded to units of
// 2^-72, so that the total does not depend on the order of the additions.  The rest
// is at most 2^31 units either way: its word takes 2^32 additions before it could
// overflow.  An atom of a cell of one atom with N neighbours gets about N^2 / 4 of
// them (fcc Cu: 2.6e6 at a three-body cutoff of 40 Bohr, 3.0e7 at 60, 2^32 at 135),
// an atom of a larger cell fewer.  Sums reach to +-2^23.  A value of 2^22 or more, an
// infinity or a NaN has no such form: the caller marks the tile (fixed_fits).
__device__ __forceinline__ void fixed_split(double v, long long& hi, long long& lo)
{
    const double sv = v * 1099511627776.0;              // 2^40
    const double h = rint(sv);
    hi = (long long)h;
    lo = __double2ll_rn((sv - h) * 4294967296.0);       // 2^32
}

__device__ __forceinline__ bool fixed_fits(long long hi)
{
    return (unsigned long long)(hi + (1LL << 62)) < (1ULL << 63);
}

// Sums of a three-body tile: energy, the nine sums of F (x) T, two words each, and the
// mark that a sum of the tile or of its atoms met a value without fixed-point form:
// the results it enters are NaN.
constexpr int kTileSums = kAtmTileSums, kTileMark = kAtmTileSums - 1;

__device__ __forceinline__ double fixed_value(const unsigned long long* acc2)
{
    return double((long long)acc2[0]) * 9.094947017729282e-13 +       // 2^-40
           double((long long)acc2[1]) * 2.117582368135751e-22;        // 2^-72
}

}  // namespace
}  // namespace d3
