// Terms of the two-body sum shared by the pair kernels (d3_pair_tt.cu,
// d3_molecule.cu): the smooth cutoff and the damping families.
#pragma once

#include "d3_device.cuh"
#include "d3_math.cuh"

namespace d3 {

template <class R> __device__ __forceinline__ R tt_sqrt(R x) { if constexpr (sizeof(R) == 8) return sqrt(x); else return sqrtf(x); }
template <class R> __device__ __forceinline__ R tt_pow(R x, R a) { if constexpr (sizeof(R) == 8) return pow(x, a); else return powf(x, a); }

template <class R>
__device__ __forceinline__ void tt_smooth(R r, R cutoff, R width, R& sw, R& dswdr)
{
    // cutoff.f90:73-99
    if (width <= R(0) || width >= cutoff) { sw = R(1); dswdr = R(0); return; }
    const R inner = cutoff - width;
    if (r <= inner) { sw = R(1); dswdr = R(0); }
    else if (r >= cutoff) { sw = R(0); dswdr = R(0); }
    else {
        const R x = (cutoff - r) / width;
        sw = x * x * x * (R(10) + x * (R(-15) + R(6) * x));
        dswdr = R(-30) * x * x * (R(1) - x) * (R(1) - x) / width;
    }
}

// One (i, j, T) term of the modified zero, optimized power, CSO and Z forms:
// edisp0 and gdisp0 as the reference names them (E = -C6 edisp0 / 2 per
// half, gradient -C6 gdisp0 v) and, for Z damping, cdisp0 = d(C6 edisp0)/dC6.
// r1 is the distance when the smooth cutoff computed it.  Pair constants:
//   kMZero:          q1 = 1/(rs6 R0), q2 = 1/(rs8 R0), q3 = bet R0,
//                    q4 = rs6 bet R0^2, q5 = rs8 bet R0^2       (mzero.f90:441-472)
//   kOptimizedPower: q1 = R0^bet R0^6, q2 = R0^bet R0^8         (optimizedpower.f90:421-448)
//   kCSO:            q1 = (a3 sqrt(rrij) + a4)^6, q2 = a2 sqrt(rrij) (cso.f90:421-446)
//   kZDamping:       zc = a1 C6 / (species index sum)          (z.f90:412-431)
// The optimized power terms use r^-bet in place of the reference's
// r^bet / (r^bet r^6 + ...) and the CSO derivative 1 - sf = ef sf in the
// FP32 form, so that no intermediate leaves the FP32 range.
template <class R, int DAMP>
__device__ __forceinline__ void tt_family(R r2, R r1, bool have_r1, R rrij, R q1, R q2, R q3, R q4, R q5, R zc,
                                          R s6, R s8, R alp6, R alp8, R bet, R a1, int h6, int hb, R& edisp0,
                                          R& gdisp0, R& cdisp0)
{
    if constexpr (DAMP == kMZero) {
        if (!have_r1) r1 = tt_sqrt<R>(r2);
        const R ir2 = inv<R>(r2);
        const R ir6 = ir2 * ir2 * ir2;
        const R x6 = inv<R>(r1 * q1 + q3), x8 = inv<R>(r1 * q2 + q3);
        const R t6 = damping_power(h6 >= 0 ? ipow(x6 * x6, h6) : tt_pow<R>(x6, alp6));
        const R t8 = damping_power(h6 >= 0 ? ipow(x8 * x8, h6 + 1) : tt_pow<R>(x8, alp8));
        const R f6 = inv<R>(R(1) + R(6) * t6);
        const R f8 = inv<R>(R(1) + R(6) * t8);
        const R d6 = R(-6) * f6 * ir2 + R(6) * alp6 * t6 * (f6 * f6) * inv<R>(r2 + q4 * r1);
        const R d8 = R(-8) * f8 * ir2 + R(6) * alp8 * t8 * (f8 * f8) * inv<R>(r2 + q5 * r1);
        const R c6 = s6 * ir6, c8 = s8 * rrij * (ir6 * ir2);
        edisp0 = c6 * f6 + c8 * f8;
        gdisp0 = c6 * d6 + c8 * d8;
    } else if constexpr (DAMP == kOptimizedPower) {
        // t6 = r^b / (r^b r^6 + q1) = 1 / (r^6 + q1 r^-b)
        const R ir2 = inv<R>(r2);
        const R ib = damping_power(hb >= 0 ? ipow(ir2, hb) : tt_pow<R>(r2, R(-0.5) * bet));
        const R r4 = r2 * r2;
        const R t6 = inv<R>(r4 * r2 + q1 * ib);
        const R t8 = inv<R>(r4 * r4 + q2 * ib);
        const R d6 = R(-6) * r4 * t6 * t6 + bet * q1 * t6 * t6 * ib * ir2;
        const R d8 = R(-8) * r4 * r2 * t8 * t8 + bet * q2 * t8 * t8 * ib * ir2;
        edisp0 = s6 * t6 + s8 * rrij * t8;
        gdisp0 = s6 * d6 + s8 * rrij * d8;
    } else if constexpr (DAMP == kCSO) {
        if (!have_r1) r1 = tt_sqrt<R>(r2);
        R sf, om;
        if constexpr (sizeof(R) == 8) {
            const R ef = exp(r1 - q2);
            sf = R(1) / (R(1) + ef);
            om = R(1) - sf;
        } else {
            const R ef = expf(fminf(r1 - q2, 80.f));
            sf = R(1) / (R(1) + ef);
            om = ef * sf;
        }
        const R sig = s6 + a1 * sf;
        const R r4 = r2 * r2;
        const R t6 = inv<R>(r4 * r2 + q1);
        const R dsig = -a1 * sf * om / r1;
        const R dt6 = R(-6) * r4 * t6 * t6;
        edisp0 = sig * t6;
        gdisp0 = dsig * t6 + sig * dt6;
    } else {
        const R r4 = r2 * r2;
        const R r6 = r4 * r2, r8 = r4 * r4;
        const R t6 = inv<R>(r6 + zc);
        const R t8 = inv<R>(r8 + zc * rrij);
        const R s8rr = s8 * rrij;
        edisp0 = s6 * t6 + s8rr * t8;
        gdisp0 = R(-6) * s6 * (r4 * t6) * t6 + R(-8) * s8rr * (r4 * r2 * t8) * t8;
        cdisp0 = s6 * (r6 * t6) * t6 + s8rr * (r8 * t8) * t8;
    }
}

}  // namespace d3
