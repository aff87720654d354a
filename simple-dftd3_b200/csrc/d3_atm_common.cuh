// Smooth cutoff and triple ownership of the three-body kernels (d3_atm.cu) and
// of the pairwise decomposition (d3_pairwise.cu).
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

}  // namespace
}  // namespace d3
