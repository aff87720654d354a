// Axilrod-Teller-Muto three-body dispersion (get_atm_dispersion, atm.f90:433-825)
// with energy, gradient, virial and dE/dCN, for molecules and periodic systems.
//
// Pair form.  With x = r^2 of the three pairs of a triple, u = 1/x,
// m = sqrt(C6) r^-3 (times the smooth switch of the pair) and P = (r0/r)^(alp/3)
// every factor of the triple is a product of pair factors:
//   E = s9 M (1 + A) f,  M = m m m,  A = 3/8 S u u u,  f = 1 / (1 + 6 P P P),
//   S = (x1 + x3 - x2)(x1 + x2 - x3)(x2 + x3 - x1)          (atm.f90:744-776)
// and with K = (1 + A)(alp/2 6P f - 3/2) - A (P the product; alp = (alp + 2)/3)
//   dE/dx1 = M f (u1 K + 3/8 u u u dS/dx1).
// So the triple loop reads one 4-value record per pair and adds to two sums per
// pair, D = sum dE/dx and W = sum E: gradient (2 D v), virial, dE/dCN
// (W/2 dlnC6/dCN) and the derivative of the switch (W dln(sw)/dx) follow from D
// and W once per pair instead of once per triple, and a pair outside the cutoff,
// a ghost or a padding slot is a record with m = 0: the loop has no tests.
//
// Tiles and blocks.  Every 32-atom tile of the spatial order is cut into compact
// tiles of 8 atoms (k_atm_order).  A block holds the 64 records of a tile pair
// (A, B <= A) for one lattice translation (k_atm_pairs; batches whose blocks
// exceed kAtmDenseCap keep only those whose spheres are in reach, k_atm_mark, and
// above kAtmGroupCands candidates take groups of systems one after the other).
// Tiles of 8 fill 0.6 of their triple slots with accepted triples on periodic
// frames (cutoff 40 Bohr), tiles of 16 0.44 and of 32 0.30 (CPU replay).
//
// Triples (k_atm_triples).  Every unordered triple of tile images (modulo a
// common translation) is visited once.  A unit is a pair block (J, K, T) whose
// third atoms, the roots, run over the tiles I > J and their images; for J = K
// (T in one half space, T = 0 as half of the walk) over all tiles, and then the
// triples inside one tile index are met three times and weighted by 1/3
// (k_atm_lists: the tile images in reach of J).  One warp takes a unit: four
// quarters of eight lanes hold four roots, the lane one atom j, its eight (j, k)
// records and their sums D, W in registers, and the quarter walks
// k = (j + t) mod 8; the sums of (i, k) move one lane down per step with k.  Roots
// without a partner in J or K inside the cutoff are dropped before (8-bit masks of
// the blocks).  Per four roots D and W of (i, j) and (i, k) become forces; every
// 128 roots the (j, k) sums do.
//
// All sums over units go to fixed-point accumulators (integer additions), so the
// results do not depend on the order of the warps and repeat bit for bit.
#include <cub/cub.cuh>
#include <math_constants.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "d3_atm_common.cuh"
#include "d3_device.cuh"
#include "d3_math.cuh"
#include "d3_per_device.h"

namespace d3 {

namespace {

constexpr int kT8 = 8;                  // atoms per three-body tile
constexpr int kRecs = kT8 * kT8;        // records per block
constexpr int kAtmWarps = 4;            // warps per block of the triple kernel
constexpr int kRing = 512;              // root queue of a warp: up to 127 left over + 32 tiles of 8
constexpr int kRootChunk = 128;         // roots between two flushes: FP32 sums run over at most 32 terms

// Resident blocks per SM the triple kernel is compiled for.  FP32 with gradient:
// 168 registers and 12 warps beat 128 registers (spills) and 16 warps, 54.8
// against 59.1 ms on eight frames; FP64 with gradient: 252 registers and 8 warps
// beat 168 and 12 (cluster of 5000 atoms 15.5 against 17.7 ms); energies: 16 and
// 12 warps beat 20 and 16 (slab 0.63 against 0.74 ms, before its pair sweeps were
// cut into more items).
template <class R, bool GRAD>
constexpr int kTripleBlocks = sizeof(R) == 4 ? (GRAD ? 3 : 4) : (GRAD ? 2 : 3);

template <class R> struct RecT;
template <> struct RecT<double> { using rec = double4; using aux = double2; };
template <> struct RecT<float> { using rec = float4; using aux = float2; };

__device__ __forceinline__ bool in_shell(double r2, double cut2) { return !(r2 > cut2 || r2 < DBL_EPSILON); }

__device__ __forceinline__ double norm2(double x, double y, double z)
{
    return __fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)));
}

__device__ __forceinline__ void fixed_add(unsigned long long* acc2, double v, unsigned long long* tile)
{
    long long hi, lo;
    fixed_split(v, hi, lo);
    if (!fixed_fits(hi)) tile[kTileMark] = 1;
    atomicAdd(acc2, (unsigned long long)hi);
    atomicAdd(acc2 + 1, (unsigned long long)lo);
}

// Two values worked on together: the packed FP32 instructions of sm_100 (one
// issue slot for two operations), or a plain pair in FP64.
struct F2 { unsigned long long v; };
struct D2 { double a, b; };
template <class R> struct PairT;
template <> struct PairT<float> { using type = F2; };
template <> struct PairT<double> { using type = D2; };

__device__ __forceinline__ F2 pk(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ D2 pk(double a, double b) { return D2{a, b}; }
__device__ __forceinline__ float lo(F2 x) { return __uint_as_float((unsigned)x.v); }
__device__ __forceinline__ float hi(F2 x) { return __uint_as_float((unsigned)(x.v >> 32)); }
__device__ __forceinline__ double lo(D2 x) { return x.a; }
__device__ __forceinline__ double hi(D2 x) { return x.b; }
__device__ __forceinline__ F2 operator+(F2 x, F2 y)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 x, F2 y)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 x, F2 y)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ F2 fma(F2 x, F2 y, F2 z)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(x.v), "l"(y.v), "l"(z.v));
    return r;
}
__device__ __forceinline__ D2 operator+(D2 x, D2 y) { return D2{x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ D2 operator-(D2 x, D2 y) { return D2{x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ D2 operator*(D2 x, D2 y) { return D2{x.a * y.a, x.b * y.b}; }
__device__ __forceinline__ D2 fma(D2 x, D2 y, D2 z) { return D2{::fma(x.a, y.a, z.a), ::fma(x.b, y.b, z.b)}; }

// Candidate block c of the processing order: system, tile pair (A >= B, local
// tile indices) and translation index.
struct BlockId { int sys, t8, A, B, t; };

// Largest a with a (a + 1) / 2 <= p.
__device__ __forceinline__ int triangle_row(unsigned p)
{
    int a = (int)((sqrtf(8.0f * (float)p + 1.0f) - 1.0f) * 0.5f);
    while ((unsigned)(a + 1) * (unsigned)(a + 2) / 2 <= p) a++;
    while ((unsigned)a * (unsigned)(a + 1) / 2 > p) a--;
    return a;
}

// System at candidate c: a 32-way search by the whole warp; returns its position.
__device__ __forceinline__ int find_system(const AtmView& v, long long c, int lane)
{
    int lo = 0, hi = v.nord;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5;
        const int p = lo + lane * step;
        const unsigned ok = __ballot_sync(0xffffffffu, p < hi && v.cand_off[p] <= c);
        lo += (__popc(ok) - 1) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

__device__ __forceinline__ BlockId block_id(const AtmView& v, long long c, int lane)
{
    const int at = find_system(v, c, lane);
    BlockId id;
    id.sys = v.ord[at];
    id.t8 = v.t8_off[id.sys];
    const long long e = c - v.cand_off[at];
    const int nT = v.rep[4 * id.sys + 3];
    const unsigned p = (unsigned)(e / nT);
    id.t = (int)(e - (long long)p * nT);
    id.A = triangle_row(p);
    id.B = (int)(p - (unsigned)id.A * (unsigned)(id.A + 1) / 2);
    return id;
}

// Unit u of the triple kernel, in the order of their work: for every system first
// the pairs of a tile with itself, whose roots are all tiles, then the others by
// rising A, whose roots are the tiles above A.  Returns the candidate.
__device__ __forceinline__ long long unit_id(const AtmView& v, long long u, int lane, BlockId& id)
{
    const int at = find_system(v, u, lane);
    id.sys = v.ord[at];
    id.t8 = v.t8_off[id.sys];
    const int nt8 = v.t8_off[id.sys + 1] - id.t8, nT = v.rep[4 * id.sys + 3];
    const long long base = v.cand_off[at];
    const unsigned p = (unsigned)((u - base) / nT);
    id.t = (int)((u - base) - (long long)p * nT);
    if (p < (unsigned)nt8) {
        id.A = id.B = (int)p;
    } else {
        const unsigned r = p - (unsigned)nt8;
        id.A = triangle_row(r) + 1;
        id.B = (int)(r - (unsigned)id.A * (unsigned)(id.A - 1) / 2);
    }
    return base + ((long long)id.A * (id.A + 1) / 2 + id.B) * nT + id.t;
}

// ------------------------------------------------------------- tile order --

// Axis of the longest extent of the atoms in group g of the warp.
__device__ __forceinline__ int longest_axis(double x, double y, double z, bool mine)
{
    double lo[3] = {mine ? x : DBL_MAX, mine ? y : DBL_MAX, mine ? z : DBL_MAX};
    double hi[3] = {mine ? x : -DBL_MAX, mine ? y : -DBL_MAX, mine ? z : -DBL_MAX};
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 3; k++) {
            lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    const double ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    return ex >= ey && ex >= ez ? 0 : ey >= ez ? 1 : 2;
}

// The coordinate as an integer of the same order, NaN at the ends: ranks by it are a
// permutation for any input, so that every slot of a tile is written.
__device__ __forceinline__ long long order_bits(double c)
{
    const long long u = __double_as_longlong(c);
    return u ^ ((u >> 63) & 0x7fffffffffffffffLL);
}

// Compact tiles of 8 atoms inside each 32-atom tile (one warp each): the atoms
// are ordered along the longest axis of their box and cut into tiles of 8, above
// 16 atoms into two halves that are ordered along their own longest axis (fill
// of the triple slots on periodic frames 0.56, against 0.49 with fixed x and y).
// Also writes the tiles' positions and clears the accumulators of the evaluation.
__global__ void k_atm_order(Batch b, const int* tile_off, const int* tile_sys, int ntiles, AtmView v, double4* spheres,
                            unsigned long long* fxf, unsigned long long* fxe, unsigned long long* queue)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x < 2) queue[threadIdx.x] = 0;
    if (tile >= ntiles) return;
    const int sys = tile_sys[tile];
    const int lt = tile - tile_off[sys];
    const int a0 = b.atom_off[sys] + lt * kTile;
    const int n = min(kTile, b.atom_off[sys + 1] - a0);
    const bool in = lane < n;
    const int a = a0 + (in ? lane : 0);
    const double x = b.x[a], y = b.y[a], z = b.z[a];
    auto rank_in = [&](int axis, int group) {
        const long long c = order_bits(axis == 0 ? x : axis == 1 ? y : z);
        int r = 0;
        for (int k = 0; k < n; k++) {
            const long long ck = __shfl_sync(0xffffffffu, c, k);
            const int gk = __shfl_sync(0xffffffffu, group, k);
            r += gk == group && (ck < c || (ck == c && k < lane));
        }
        return r;
    };
    int slot = rank_in(longest_axis(x, y, z, in), 0);
    if (n > 16) {
        const int half = slot >> 4;
        const int ax0 = longest_axis(x, y, z, in && half == 0), ax1 = longest_axis(x, y, z, in && half == 1);
        slot = 16 * half + rank_in(half ? ax1 : ax0, half);
    }
    const int base8 = v.t8_off[sys] + 4 * lt;
    const int n8 = (n + kT8 - 1) / kT8;
    if (in) {
        v.sub[kT8 * base8 + slot] = a;
        v.pos[kT8 * base8 + slot] = make_double4(x, y, z, (double)a);
    } else if (lane < kT8 * n8) {
        v.sub[kT8 * base8 + lane] = -1;
        v.pos[kT8 * base8 + lane] = make_double4(0.0, 0.0, 0.0, 0.0);
    }
    if (fxf && in) {
        unsigned long long* f = fxf + (size_t)8 * a;
#pragma unroll
        for (int k = 0; k < 8; k++) f[k] = 0;
    }
    if (lane < n8) {
        unsigned long long* f = fxe + (size_t)kTileSums * (base8 + lane);
#pragma unroll
        for (int k = 0; k < kTileSums; k++) f[k] = 0;
    }
    if (!spheres) return;
    // bounding spheres (box centre, largest distance)
    for (int q = 0; q < n8; q++) {
        const bool mine = in && (slot >> 3) == q;
        double lo[3] = {mine ? x : DBL_MAX, mine ? y : DBL_MAX, mine ? z : DBL_MAX};
        double hi[3] = {mine ? x : -DBL_MAX, mine ? y : -DBL_MAX, mine ? z : -DBL_MAX};
        for (int o = 16; o > 0; o >>= 1)
            for (int k = 0; k < 3; k++) {
                lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
        double c[3], d2 = 0.0;
        for (int k = 0; k < 3; k++) c[k] = 0.5 * (lo[k] + hi[k]);
        if (mine) d2 = norm2(x - c[0], y - c[1], z - c[2]);
        for (int o = 16; o > 0; o >>= 1) d2 = fmax(d2, __shfl_xor_sync(0xffffffffu, d2, o));
        if (lane == 0) spheres[base8 + q] = make_double4(c[0], c[1], c[2], sqrt(d2));
    }
}

// ------------------------------------------------------------ pair blocks --

// flag[c] = 1 for the candidate blocks whose spheres are within the cutoff
// (with a margin far above the rounding of the sphere test).
__global__ void k_atm_mark(Batch b, Config c, AtmView v, const double4* spheres, int* flag)
{
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) & ~31LL;
    if (w0 >= v.ncand) return;
    // the 32 candidates of a warp may span systems: the search takes them one
    // system at a time only where they do
    const long long cand = w0 + lane;
    const BlockId first = block_id(v, w0, lane);
    const long long last_c = min(w0 + 31, v.ncand - 1);
    const BlockId last = block_id(v, last_c, lane);
    BlockId id = first;
    if (first.sys == last.sys) {
        const int nT = v.rep[4 * first.sys + 3];
        const long long t = (long long)first.t + lane;
        long long p = (long long)first.A * (first.A + 1) / 2 + first.B + t / nT;
        id.t = (int)(t % nT);
        int a = first.A;
        while ((long long)(a + 1) * (a + 2) / 2 <= p) a++;
        id.A = a;
        id.B = (int)(p - (long long)a * (a + 1) / 2);
    } else {
        for (int k = 0; k < 32; k++) {
            const BlockId q = block_id(v, min(w0 + k, v.ncand - 1), lane);
            if (k == lane) id = q;
        }
    }
    if (cand >= v.ncand) return;
    const double4 sa = spheres[id.t8 + id.A], sb = spheres[id.t8 + id.B];
    const double* T = b.img + 3 * (size_t)(b.img_off[kImgDisp3 * (b.nsys + 1) + id.sys] + id.t);
    const double reach = (c.cut3 + sa.w + sb.w) * (1.0 + 1e-9) + 1e-9;
    flag[cand] = norm2(sb.x + T[0] - sa.x, sb.y + T[1] - sa.y, sb.z + T[2] - sa.z) <= reach * reach ? 1 : 0;
}

__global__ void k_atm_guard(const int* total, long long cap, int* guard, bool first)
{
    *guard = *total > cap || (!first && *guard) ? 1 : 0;
}

// The 64 records {x, u, m, P} of a block and, with gradients, {dlnC6/dCN_a / 2,
// dlnC6/dCN_b / 2} of (row atom a of A, column atom b of B + T): one warp per
// candidate.  C6 is the dot product of a's reference weights with b's species
// vector for a's species, U_b[s_a][r] = sum_q C6ref(r, q) gw_b[q]
// (get_atomic_c6, model.f90:432-461).  mask: bits 0-7 the rows, bits 8-15 the
// columns with a pair inside the cutoff.
template <class R>
__global__ void __launch_bounds__(256)
k_atm_pairs(Batch b, Species s, Config c, Work w, AtmView v, const R* UV, double alp3, const int* guard)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long cand = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (cand >= v.ncand || (guard && *guard)) return;
    long long blk = cand;
    if (v.map) {
        const int m0 = v.map[cand], m1 = v.map[cand + 1];
        if (m0 == m1) {
            if (lane == 0) v.mask[cand] = 0;
            return;
        }
        blk = m0;
    }
    const BlockId id = block_id(v, cand, lane);
    const double* T = b.img + 3 * (size_t)(b.img_off[kImgDisp3 * (b.nsys + 1) + id.sys] + id.t);
    const double tx = T[0], ty = T[1], tz = T[2];
    const double cut2 = c.cut3 * c.cut3;
    const int bc = v.sub[kT8 * (id.t8 + id.B) + (lane & 7)];
    double x2[2];
    int ar[2];
    bool ok[2];
    unsigned vote[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        ar[h] = v.sub[kT8 * (id.t8 + id.A) + 4 * h + (lane >> 3)];
        x2[h] = 1.0;
        ok[h] = ar[h] >= 0 && bc >= 0;
        if (ok[h]) {
            const double r2 = norm2(b.x[bc] + tx - b.x[ar[h]], b.y[bc] + ty - b.y[ar[h]], b.z[bc] + tz - b.z[ar[h]]);
            ok[h] = in_shell(r2, cut2);
            if (ok[h]) x2[h] = r2;
        }
        vote[h] = __ballot_sync(0xffffffffu, ok[h]);
    }
    if (lane == 0) {
        unsigned rows = 0, cols = vote[0] | vote[1];
        cols |= cols >> 16;
        cols |= cols >> 8;
        for (int q = 0; q < 4; q++) {
            rows |= ((vote[0] >> (8 * q)) & 0xffu) ? 1u << q : 0u;
            rows |= ((vote[1] >> (8 * q)) & 0xffu) ? 1u << (q + 4) : 0u;
        }
        v.mask[cand] = (unsigned short)(rows | (cols & 0xffu) << 8);
    }
    if (!(vote[0] | vote[1])) return;
    using Rec = typename RecT<R>::rec;
    using Aux = typename RecT<R>::aux;
    Rec* rec = static_cast<Rec*>(v.rec) + blk * kRecs;
    Aux* aux = static_cast<Aux*>(v.aux) + blk * kRecs;
    const R* gw_all = (const R*)(sizeof(R) == 8 ? (const void*)w.gw : (const void*)w.gwf);
    const R* dgw_all = (const R*)(sizeof(R) == 8 ? (const void*)w.dgw : (const void*)w.dgwf);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        Rec o;
        o.x = R(1); o.y = R(0); o.z = R(0); o.w = R(0);
        Aux q;
        q.x = R(0); q.y = R(0);
        if (ok[h]) {
            const int a = ar[h];
            const int sa = b.sp[a], sb = b.sp[bc];
            // FP64 up to the record, whose values are rounded once each in the mixed form
            const double u = rcp_fast(x2[h]);
            o.x = R(x2[h]);
            o.y = R(u);
            const R* gw = gw_all + (size_t)a * kMaxRef;
            const R* dgw = dgw_all + (size_t)a * kMaxRef;
            const R* up = UV + ((size_t)bc * b.nid + sa) * (2 * kRefPad);
            const int nr = s.nref[sa];
            R c6 = R(0), dr = R(0), dc = R(0);
            for (int r = 0; r < nr; r++) {
                const R u0 = __ldg(up + r);
                c6 += gw[r] * u0;
                dr += dgw[r] * u0;
                dc += gw[r] * __ldg(up + kRefPad + r);
            }
            if (b.ghost && b.ghost[a]) c6 = R(0);
            const double r0 = __ldg(s.atm_r0 + sa * b.nid + sb);
            // the pair's share of (r0/r)^alp3, bounded so that the product of three (FP32:
            // of two; the third may take it to infinity, where f is zero) stays finite
            if constexpr (sizeof(R) == 8) {
                o.w = fmin(exp(0.5 * alp3 * log(r0 * r0 * u)), 1e100);
            } else {
                const double l = 0.5 * alp3 * log2(r0 * r0 * u);
                const float lh = (float)l, ll = (float)(l - (double)lh);
                const float p = exp2f(lh);
                o.w = fminf(::fma(0.69314718f * ll, p, p), 1e18f);
            }
            if (c6 != R(0)) {
                R m = R(double(sqrt(c6)) * (u * rsqrt_fast(x2[h])));
                if (c.width3 > 0.0) {
                    R sw, dsw;
                    smooth<R>(R(sqrt(x2[h])), R(c.cut3), R(c.width3), sw, dsw);
                    m *= sw;
                }
                o.z = m;
                const R ic6 = R(0.5) / c6;
                q.x = dr * ic6;
                q.y = dc * ic6;
            }
        }
        rec[32 * h + lane] = o;
        if (c.grad) aux[32 * h + lane] = q;
    }
}

// Root tiles of every tile J, ascending: the tile images (I, T_I) whose block
// with J has a pair inside the cutoff, {block, mask of the roots << 24 | I, T_I,
// candidate}.  One warp per tile; gt[J] is the first entry with I > J.
__global__ void k_atm_lists(AtmView v, int ntiles8, const int* tile8_sys, const int* sys_group, int group,
                            const long long* list_off, int4* list, int2* range, const int* guard)
{
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tile >= ntiles8 || (guard && *guard)) return;
    const int sys = tile8_sys[tile];
    if (sys_group && sys_group[sys] != group) return;
    const int t8 = v.t8_off[sys], nt8 = v.t8_off[sys + 1] - t8, J = tile - t8;
    const int nT = v.rep[4 * sys + 3];
    const long long cbase = v.cand_off_sys[sys];
    int4* out = list + list_off[sys] + (long long)J * nt8 * nT;
    int n = 0, gt = 0;
    for (int e0 = 0; e0 < nt8 * nT; e0 += 32) {
        const int e = e0 + lane;
        int4 o = make_int4(0, 0, 0, 0);
        unsigned m = 0;
        int I = 0;
        if (e < nt8 * nT) {
            I = nT == 1 ? e : e / nT;
            const int tI = e - I * nT;
            // stored as (I, J) with J at -T_I, or for I < J as (J, I) with I at T_I
            const long long c = I < J ? cbase + ((long long)J * (J + 1) / 2 + I) * nT + tI
                                      : cbase + ((long long)I * (I + 1) / 2 + J) * nT + (nT - 1 - tI);
            m = v.mask[c];
            m = I < J ? m >> 8 : m & 0xffu;
            if (m) o = make_int4((int)(v.map ? v.map[c] : c), (int)(m << 24) | I, tI, 0);
        }
        const unsigned keep = __ballot_sync(0xffffffffu, m != 0);
        gt += __popc(__ballot_sync(0xffffffffu, m != 0 && I <= J));
        if (m) out[n + __popc(keep & ((1u << lane) - 1u))] = o;
        n += __popc(keep);
    }
    if (lane == 0) range[tile] = make_int2(gt, n);
}

// ---------------------------------------------------------------- triples --

template <class R>
__device__ __forceinline__ R sel(bool p, R a, R b) { return p ? a : b; }

// dln(sw)/dx of a pair's switch at r = sqrt(x) (zero where the switch is 1 or 0)
template <class R>
__device__ __forceinline__ R dln_switch(R x, R cutoff, R width)
{
    R sw, dsw;
    const R r = sqrt(x);
    smooth<R>(r, cutoff, width, sw, dsw);
    return sw > R(0) ? R(0.5) * dsw / (sw * r) : R(0);
}

// Per-warp shared memory of the triple kernel: the records of four roots (two
// buffers, filled one step of four ahead by asynchronous copies) and the queue.
template <class R>
struct AtmStage {
    typename RecT<R>::rec ik[32], ij[32];
    typename RecT<R>::aux qij[32], qik[32];
    double4 pos[4];                  // root position, atom
    double T[4][4];                  // root translation
};
template <class R>
struct AtmShared {
    AtmStage<R> st[2];
    float4 xu[32], mp[32];           // FP32: (i, k) records of k and k ^ 4, {x, x', u, u'} and {m, m', P, P'}
    int4 ring[kRing];                // roots: first record (i, j) and (i, k), tile slot, flags and translation
    double4 pj[kT8], pk[kT8];        // positions of the atoms j and (at their image) k
};

template <int BYTES>
__device__ __forceinline__ void async_copy(void* dst, const void* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
template <class V>
__device__ __forceinline__ void async_copy_value(V* dst, const V* src)
{
    if constexpr (sizeof(V) == 32) {
        async_copy<16>(dst, src);
        async_copy<16>(reinterpret_cast<char*>(dst) + 16, reinterpret_cast<const char*>(src) + 16);
    } else {
        async_copy<(int)sizeof(V)>(dst, src);
    }
}

// Columns of the pair p of a step: with gradients the lanes of a quarter take
// different k, (j + p) mod 8 and k ^ 4, and the column sums travel with k; energies
// have no column sums, so that all lanes take the same k, p and p + 4, and its records
// are broadcast reads (141-atom slab 339 -> 305 us; with gradients the exchanges of
// the column sums cost what the reads save: eight frames 51.2 against 52.5 ms).
template <bool GRAD>
__device__ __forceinline__ int column(int j, int p) { return GRAD ? (j + p) & 7 : p; }

// What bounds it: the data pipe of L1 and shared memory (74% busy in FP32, 86% in
// FP64: the (i, k) records of a step, staged roots, shuffles of the column sums),
// with 12 or 8 warps per SM to hide its latency and that of the FMA chains (2.2 and
// 1.7 instructions per cycle and SM; FMA pipe 44%, FP64 pipe 49%).  A step of two
// partners (k and k ^ 4) is 39 packed FP32 instructions, two reciprocals, four
// shuffles and two 16-byte shared loads; the (j, k) records and sums stay in
// registers.  One partner at a time and
// plain FP32 instructions (62 per step) took 67.8 instead of 54.8 ms on eight
// frames and, in FP64, 16.7 instead of 15.3 ms on the cluster (both before the unit
// order).  Whole evaluations with the neighbour-list and block-per-molecule kernels
// that this one replaced (185 instructions per slot, exp, log and divisions per
// triple in FP64) against now: cluster of 5000 atoms (FP64) 54.0 -> 15.2 ms, 512
// molecules (FP64) 21.1 -> 2.15 ms, 4096 molecules (mixed) 13.5 -> 5.9 ms, eight
// periodic frames (mixed) 166 -> 53 ms, one molecule of 100 atoms 222 -> 70 us, slab
// energy 2.73 -> 0.31 ms.
// GEN: work partition and term counting (the owner test of every triple).
template <class R, bool GRAD, bool PER, bool GEN>
__global__ void __launch_bounds__(32 * kAtmWarps, kTripleBlocks<R, GRAD>)
k_atm_triples(Batch b, Config c, Partition part, AtmView v, double alp3d, int split, int grab,
              unsigned long long* queue, unsigned long long* fxf, unsigned long long* fxe, int counting,
              const int* guard)
{
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Rec = typename RecT<R>::rec;
    using Aux = typename RecT<R>::aux;
    using Pair = typename PairT<R>::type;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    AtmShared<R>& sh = reinterpret_cast<AtmShared<R>*>(smem_raw)[wid];
    if (guard && *guard) return;                 // blocks did not fit the reserved buffers
    const Rec* rec = static_cast<const Rec*>(v.rec);
    const Aux* aux = static_cast<const Aux*>(v.aux);
    const int q = lane >> 3, j = lane & 7, qbase = lane & 24;
    const Pair ahalf = pk(R(0.5 * alp3d), R(0.5 * alp3d));
    const bool smooth_on = c.width3 > 0.0 && c.width3 < c.cut3;
    const R cutoff = R(c.cut3), width = R(c.width3);
    const unsigned long long nunits = (unsigned long long)v.ncand * split;
    unsigned long long u = 0, u_end = 0;
    for (;;) {
        if (u == u_end) {
            if (lane == 0) u = atomicAdd(queue, (unsigned long long)grab);
            u = __shfl_sync(kAll, u, 0);
            if (u >= nunits) break;
            u_end = min(u + grab, nunits);
        }
        BlockId id;
        const long long cand = unit_id(v, (long long)(u / split), lane, id);
        const int piece = (int)(u % split);
        u++;
        if (v.mask[cand] == 0) continue;
        const int nT = PER ? v.rep[4 * id.sys + 3] : 1;
        const bool same = id.A == id.B;
        if (PER && same && 2 * id.t < nT - 1) continue;      // the other half space
        const bool diag = same && 2 * id.t == nT - 1;
        const int nt8 = v.t8_off[id.sys + 1] - id.t8;
        const int J = id.A, K = id.B;
        int rx = 0, ry = 0, rz = 0, jx = 0, jy = 0, jz = 0;
        if (PER) {
            rx = v.rep[4 * id.sys]; ry = v.rep[4 * id.sys + 1]; rz = v.rep[4 * id.sys + 2];
            jz = id.t % (2 * rz + 1) - rz;
            jy = id.t / (2 * rz + 1) % (2 * ry + 1) - ry;
            jx = id.t / ((2 * rz + 1) * (2 * ry + 1)) - rx;
        }
        const long long cbase = cand - ((long long)J * (J + 1) / 2 + K) * nT - id.t;    // first candidate of the system
        const double* img = b.img + 3 * (size_t)b.img_off[kImgDisp3 * (b.nsys + 1) + id.sys];
        const double kx = PER ? img[3 * id.t] : 0.0, ky = PER ? img[3 * id.t + 1] : 0.0,
                     kz = PER ? img[3 * id.t + 2] : 0.0;
        const long long bjk = v.map ? v.map[cand] : cand;
        const int aj = v.sub[kT8 * (id.t8 + J) + j], ak = v.sub[kT8 * (id.t8 + K) + j];
        if (GRAD && q < 2) {
            double4 o = v.pos[kT8 * (id.t8 + (q ? K : J)) + j];
            if (q) { o.x += kx; o.y += ky; o.z += kz; }
            (q ? sh.pk : sh.pj)[j] = o;
        }
        __syncwarp();
        int oj = 0, ok = 0;
        if (GEN) {
            oj = aj >= 0 ? b.local[aj] : 0;
            ok = ak >= 0 ? b.local[ak] : 0;
        }
        // the (j, k) records of this lane; pair p: k = column(j, p) and k ^ 4.  A tile
        // with itself (diag): every unordered pair once.
        Pair zx[4], zu[4], zm[4], zp[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int k0 = column<GRAD>(j, p);
            Rec r0 = rec[bjk * kRecs + kT8 * j + k0], r1 = rec[bjk * kRecs + kT8 * j + (k0 ^ 4)];
            if (diag) {
                // the rotated walk takes steps 1..3, and 4 in the lower lanes
                if (GRAD ? p == 0 : k0 >= j) { r0.z = R(0); if (GEN) r0.y = R(0); }
                if (GRAD ? p > 0 || j >= 4 : k0 + 4 >= j) { r1.z = R(0); if (GEN) r1.y = R(0); }
            }
            zx[p] = pk(r0.x, r1.x); zu[p] = pk(r0.y, r1.y); zm[p] = pk(r0.z, r1.z); zp[p] = pk(r0.w, r1.w);
        }
        // root tiles from the lists of J, or (one lattice point, no lists) all tiles
        const int4* list = nullptr;
        int nE = nt8, e0 = (same ? 0 : J + 1) + piece;
        if (PER || v.list) {
            const int2 range = v.range[id.t8 + J];
            list = v.list + v.list_off[id.sys] + (long long)J * nt8 * nT;
            nE = range.y;
            e0 = (same ? 0 : range.x) + piece;
        }
        int head = 0, cnt = 0;
        while (true) {
            // roots: tiles I (and images) with a pair in reach of both J and K
            while (cnt < kRootChunk && e0 < nE) {
                const int e = e0 + lane * split;
                e0 += 32 * split;
                unsigned m = 0;
                int bij = 0, bik = 0, I = 0, fl = 0;
                if (e < nE) {
                    int tI = 0;
                    unsigned mij;
                    if (PER || list) {
                        const int4 en = list[e];
                        bij = en.x;
                        I = en.y & 0xffffff;
                        mij = (unsigned)en.y >> 24;
                        tI = en.z;
                    } else {
                        I = e;
                        bij = (int)(I < J ? cbase + (long long)J * (J + 1) / 2 + I : cbase + (long long)I * (I + 1) / 2 + J);
                        mij = v.mask[bij];
                        mij = I < J ? mij >> 8 : mij & 0xffu;
                    }
                    int d = 0;
                    bool in = true;
                    const bool tr = I < J;                  // block stored as (J, I)
                    if (PER) {
                        const int iz = tI % (2 * rz + 1) - rz, iy = tI / (2 * rz + 1) % (2 * ry + 1) - ry,
                                  ix = tI / ((2 * rz + 1) * (2 * ry + 1)) - rx;
                        // translation of K seen from the root: T - T_I (of the root seen from K: T_I - T)
                        const int sg = tr ? -1 : 1;
                        const int dx = sg * (jx - ix), dy = sg * (jy - iy), dz = sg * (jz - iz);
                        in = abs(dx) <= rx && abs(dy) <= ry && abs(dz) <= rz;
                        d = ((dx + rx) * (2 * ry + 1) + (dy + ry)) * (2 * rz + 1) + dz + rz;
                    }
                    if (in) {
                        const long long cik = tr ? cbase + ((long long)J * (J + 1) / 2 + I) * nT + d
                                                 : cbase + ((long long)I * (I + 1) / 2 + K) * nT + d;
                        m = v.mask[cik];
                        m = mij & (tr ? m >> 8 : m & 0xffu);
                        if (m) bik = (int)(v.map ? v.map[cik] : cik);
                        fl = (tr ? 1 : 0) | (same && I == J ? 2 : 0) | tI << 2;
                    }
                }
                int at = __popc(m);
                int total = at;
                {
                    // exclusive prefix of the root counts
                    for (int o = 1; o < 32; o <<= 1) {
                        const int x = __shfl_up_sync(kAll, total, o);
                        if (lane >= o) total += x;
                    }
                    at = total - at;
                    total = __shfl_sync(kAll, total, 31);
                }
                if (m) {
                    const unsigned rij0 = (unsigned)bij * kRecs, rik0 = (unsigned)bik * kRecs;
                    int p = head + cnt + at;
                    while (m) {
                        const int i = __ffs(m) - 1;
                        m &= m - 1;
                        const unsigned first = (fl & 1) ? i : kT8 * i;
                        sh.ring[p & (kRing - 1)] = make_int4((int)(rij0 + first), (int)(rik0 + first), kT8 * (id.t8 + I) + i, fl);
                        p++;
                    }
                }
                cnt += total;
            }
            __syncwarp();
            if (cnt == 0) break;
            const int nroot = min(cnt, kRootChunk);
            Pair Djk[4], Wjk[4];
            Pair fjk[4];                       // force and dE/dCN of j and of k
            double vr[3] = {0, 0, 0};          // component (lane >> 1) & 3 of sum F_i (x) T_I
            double esum = 0.0;
            int ntrip = 0;
            if (GRAD)
#pragma unroll
                for (int p = 0; p < 4; p++) { Djk[p] = pk(R(0), R(0)); Wjk[p] = pk(R(0), R(0)); fjk[p] = pk(R(0), R(0)); }
            auto fetch = [&](int r0) {
                const int4 e = sh.ring[(head + min(r0 + q, nroot - 1)) & (kRing - 1)];
                AtmStage<R>& s = sh.st[(r0 >> 2) & 1];
                const unsigned step = (e.w & 1) ? kT8 * j : j;
                async_copy_value(&s.ij[lane], rec + ((unsigned)e.x + step));
                async_copy_value(&s.ik[lane], rec + ((unsigned)e.y + step));
                if (GRAD) {
                    async_copy_value(&s.qij[lane], aux + ((unsigned)e.x + step));
                    async_copy_value(&s.qik[lane], aux + ((unsigned)e.y + step));
                    if (j < 2) async_copy<16>(reinterpret_cast<char*>(&s.pos[q]) + 16 * j,
                                              reinterpret_cast<const char*>(v.pos + e.z) + 16 * j);
                    else if (PER && j < 5) async_copy<8>(&s.T[q][j - 2], img + 3 * (e.w >> 2) + j - 2);
                }
            };
            fetch(0);
            asm volatile("cp.async.commit_group;" ::: "memory");
            for (int r0 = 0; r0 < nroot; r0 += 4) {
                const bool rin = r0 + q < nroot;
                if (r0 + 4 < nroot) fetch(r0 + 4);
                asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
                __syncwarp();
                const AtmStage<R>& st = sh.st[(r0 >> 2) & 1];
                const int4 e = sh.ring[(head + min(r0 + q, nroot - 1)) & (kRing - 1)];
                Rec rij = st.ij[lane];
                int ai = 0;
                if (GEN) ai = v.sub[e.z];
                if (!rin) { rij.z = R(0); if (GEN) rij.y = R(0); }
                if (same && (e.w & 2)) rij.z *= R(1.0 / 3.0);
                if constexpr (sizeof(R) == 4) {
                    const float4 own = st.ik[lane];
                    sh.xu[lane] = make_float4(own.x, __shfl_xor_sync(kAll, own.x, 4), own.y, __shfl_xor_sync(kAll, own.y, 4));
                    sh.mp[lane] = make_float4(own.z, __shfl_xor_sync(kAll, own.z, 4), own.w, __shfl_xor_sync(kAll, own.w, 4));
                    __syncwarp();
                }
                const Pair x = pk(rij.x, rij.x), xm = pk(rij.z, rij.z), one = pk(R(1), R(1));
                const Pair xu = pk(R(0.375) * rij.y, R(0.375) * rij.y), xp = pk(R(6) * rij.w, R(6) * rij.w);
                Pair rK = pk(R(0), R(0)), rV = rK, rE = rK, kS = rK, kE = rK;
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const int kl = qbase | column<GRAD>(j, p);
                    Pair y, yu, ym, yp;
                    if constexpr (sizeof(R) == 4) {
                        const float4 b0 = sh.xu[kl], b1 = sh.mp[kl];
                        y = pk(b0.x, b0.y); yu = pk(b0.z, b0.w); ym = pk(b1.x, b1.y); yp = pk(b1.z, b1.w);
                    } else {
                        const Rec b0 = st.ik[kl], b1 = st.ik[kl ^ 4];
                        y = pk(b0.x, b1.x); yu = pk(b0.y, b1.y); ym = pk(b0.z, b1.z); yp = pk(b0.w, b1.w);
                    }
                    Pair M = xm * ym * zm[p];
                    if (GEN) {
                        R mh[2] = {lo(M), hi(M)};
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int okt = __shfl_sync(kAll, ok, kl ^ (4 * h)), akt = __shfl_sync(kAll, ak, kl ^ (4 * h));
                            bool valid = rij.y * (h ? hi(yu) * hi(zu[p]) : lo(yu) * lo(zu[p])) != R(0);
                            if (part.nparts > 1) {
                                // owner of the triple: the pair of its two largest input indices
                                int o1 = b.local[ai], o2 = oj, o3 = okt, w_;
                                if (o2 > o1) { w_ = o1; o1 = o2; o2 = w_; }
                                if (o3 > o2) { w_ = o2; o2 = o3; o3 = w_; }
                                if (o2 > o1) { w_ = o1; o1 = o2; o2 = w_; }
                                valid = valid && owns_pair_atm(part, o1, o2);
                            }
                            if (!valid) mh[h] = R(0);
                            // visits of the reference's loop (atm.f90:705-733), times three
                            const int eq = (ai == aj) + (ai == akt) + (aj == akt);
                            const int mult = eq == 3 ? 6 : eq ? 2 : 1;
                            if (valid) ntrip += (e.w & 2) ? mult : 3 * mult;
                        }
                        M = pk(mh[0], mh[1]);
                    }
                    const Pair z = zx[p];
                    const Pair U = xu * yu * zu[p];
                    const Pair p6 = xp * yp * zp[p];
                    const Pair s = x + y, d = x - y;
                    const Pair a1 = z + d, a2 = s - z, a3 = z - d;
                    const Pair q1 = a1 * a2;
                    const Pair A = q1 * a3 * U;
                    const Pair t = p6 + one;
                    const Pair f = pk(rcp_fast(lo(t)), rcp_fast(hi(t)));
                    const Pair B1 = A + one;
                    const Pair Mf = M * f;
                    if constexpr (!GRAD) {
                        rE = fma(Mf, B1, rE);
                    } else {
                        const Pair E = Mf * B1;
                        const Pair q2 = a2 * a3, q3 = a1 * a3;
                        // K = (1 + A) w - A with w = alp/2 6Pf - 3/2: (1 + A)(w - 1) + 1, 6Pf = 1 - f
                        const Pair KM = fma(B1, fma(one - f, ahalf, pk(R(-2.5), R(-2.5))), one) * Mf;
                        const Pair V = U * Mf;
                        const Pair dq = q2 - q1, sq = q2 + q1;
                        rK = rK + KM;
                        rV = fma(V, q3 + dq, rV);
                        kS = fma(yu, KM, kS);
                        kS = fma(V, q3 - dq, kS);
                        Djk[p] = fma(zu[p], KM, Djk[p]);
                        Djk[p] = fma(V, sq - q3, Djk[p]);
                        rE = rE + E;
                        kE = kE + E;
                        Wjk[p] = Wjk[p] + E;
                        // the sums of (i, k) move one lane down, with k
                        const int from = qbase | ((j + 1) & 7);
                        kS = pk(__shfl_sync(kAll, lo(kS), from), __shfl_sync(kAll, hi(kS), from));
                        kE = pk(__shfl_sync(kAll, lo(kE), from), __shfl_sync(kAll, hi(kE), from));
                    }
                }
                const R sumE = lo(rE) + hi(rE);
                esum += double(sumE);
                if constexpr (GRAD) {
                    // after four moves the lane holds column j (upper value) and column j ^ 4 (lower)
                    const R Wik = hi(kE) + __shfl_xor_sync(kAll, lo(kE), 4);
                    R Dik = hi(kS) + __shfl_xor_sync(kAll, lo(kS), 4);
                    R Dij = ::fma(rij.y, lo(rK) + hi(rK), lo(rV) + hi(rV));
                    if (smooth_on) {
                        if (sumE != R(0)) Dij += sumE * dln_switch<R>(rij.x, cutoff, width);
                        if (Wik != R(0)) Dik += Wik * dln_switch<R>(st.ik[lane].x, cutoff, width);
                    }
                    const double4 pi = st.pos[q];
                    double tix = 0, tiy = 0, tiz = 0;
                    if (PER) { tix = st.T[q][0]; tiy = st.T[q][1]; tiz = st.T[q][2]; }
                    const double xi = pi.x + tix, yi = pi.y + tiy, zi = pi.z + tiz;
                    const Aux qij = st.qij[lane], qik = st.qik[lane];
                    const bool tr = e.w & 1;
                    R g0, g1, g2, g3;
                    {
                        const double4 pj = sh.pj[j], pk_ = sh.pk[j];
                        const Pair D = pk(Dij, Dik);
                        const Pair gx = D * pk(R(pj.x - xi), R(pk_.x - xi)), gy = D * pk(R(pj.y - yi), R(pk_.y - yi)),
                                   gz = D * pk(R(pj.z - zi), R(pk_.z - zi));
                        fjk[0] = fjk[0] + gx; fjk[1] = fjk[1] + gy; fjk[2] = fjk[2] + gz;
                        fjk[3] = fma(pk(sumE, Wik), tr ? pk(qij.x, qik.x) : pk(qij.y, qik.y), fjk[3]);
                        g0 = -(lo(gx) + hi(gx)); g1 = -(lo(gy) + hi(gy)); g2 = -(lo(gz) + hi(gz));
                        g3 = ::fma(sumE, tr ? qij.y : qij.x, Wik * (tr ? qik.y : qik.x));
                    }
                    // force (and dE/dCN) of the root: component (lane >> 1) & 3 summed over the quarter
                    {
                        const bool b2 = lane & 4, b1 = lane & 2;
                        R k0 = sel(b2, g2, g0) + __shfl_xor_sync(kAll, sel(b2, g0, g2), 4);
                        R k1 = sel(b2, g3, g1) + __shfl_xor_sync(kAll, sel(b2, g1, g3), 4);
                        R kk = sel(b1, k1, k0) + __shfl_xor_sync(kAll, sel(b1, k0, k1), 2);
                        kk += __shfl_xor_sync(kAll, kk, 1);
                        const int comp = (lane >> 1) & 3;
                        const double g = double(kk);
                        if (PER) { vr[0] = ::fma(g, tix, vr[0]); vr[1] = ::fma(g, tiy, vr[1]); vr[2] = ::fma(g, tiz, vr[2]); }
                        if (rin) {
                            long long hi, lo;
                            fixed_split(g, hi, lo);
                            if (!fixed_fits(hi)) fxe[(size_t)kTileSums * (e.z >> 3) + kTileMark] = 1;
                            atomicAdd(fxf + (size_t)8 * (int)pi.w + 2 * comp + (lane & 1),
                                      (unsigned long long)((lane & 1) ? lo : hi));
                        }
                    }
                }
                __syncwarp();       // the buffer is filled again two steps on
            }
            head = (head + nroot) & (kRing - 1);
            cnt -= nroot;
            // ---- flush: energy, then the (j, k) sums and the forces of j and k
            unsigned long long* fe = fxe + (size_t)kTileSums * (id.t8 + J);
            {
                double es = esum;
                for (int o = 16; o > 0; o >>= 1) es += __shfl_xor_sync(kAll, es, o);
                if (lane == 0) fixed_add(fe, es, fe);
                if (GEN && counting) {
                    for (int o = 16; o > 0; o >>= 1) ntrip += __shfl_xor_sync(kAll, ntrip, o);
                    if (lane == 0) atomicAdd(queue + 1, (unsigned long long)ntrip);
                }
            }
            if constexpr (GRAD) {
                R fj[4], fk[4];
#pragma unroll
                for (int d = 0; d < 4; d++) { fj[d] = lo(fjk[d]); fk[d] = hi(fjk[d]); }
                // quarter q keeps the steps t = q and q + 4, summed over the quarters
                R Dt[2], Wt[2];
                {
                    // pair p holds the steps p and p + 4: halving over the quarters leaves pair q
                    const bool h16 = lane & 16, h8 = lane & 8;
                    auto halve = [&](const Pair* X, R& first, R& second) {
                        R a0[2], a1[2];
#pragma unroll
                        for (int p = 0; p < 2; p++) {
                            a0[p] = sel(h16, lo(X[p + 2]), lo(X[p])) + __shfl_xor_sync(kAll, sel(h16, lo(X[p]), lo(X[p + 2])), 16);
                            a1[p] = sel(h16, hi(X[p + 2]), hi(X[p])) + __shfl_xor_sync(kAll, sel(h16, hi(X[p]), hi(X[p + 2])), 16);
                        }
                        first = sel(h8, a0[1], a0[0]) + __shfl_xor_sync(kAll, sel(h8, a0[0], a0[1]), 8);
                        second = sel(h8, a1[1], a1[0]) + __shfl_xor_sync(kAll, sel(h8, a1[0], a1[1]), 8);
                    };
                    halve(Djk, Dt[0], Dt[1]);
                    halve(Wjk, Wt[0], Wt[1]);
                }
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const int t = q + 4 * p;
                    const int kl = qbase | ((j + t) & 7), back = qbase | ((j - t) & 7);
                    if (smooth_on && Wt[p] != R(0))
                        Dt[p] += Wt[p] * dln_switch<R>(rec[bjk * kRecs + kT8 * j + ((j + t) & 7)].x, cutoff, width);
                    const double4 pj = sh.pj[j], pk_ = sh.pk[kl & 7];
                    const R gx = Dt[p] * R(pk_.x - pj.x), gy = Dt[p] * R(pk_.y - pj.y), gz = Dt[p] * R(pk_.z - pj.z);
                    const Aux qa = aux[bjk * kRecs + kT8 * j + ((j + t) & 7)];
                    fj[0] -= gx; fj[1] -= gy; fj[2] -= gz;
                    fj[3] = ::fma(Wt[p], qa.x, fj[3]);
                    fk[0] += __shfl_sync(kAll, gx, back);
                    fk[1] += __shfl_sync(kAll, gy, back);
                    fk[2] += __shfl_sync(kAll, gz, back);
                    fk[3] += __shfl_sync(kAll, Wt[p] * qa.y, back);
                }
                // quarter q keeps component q of j and of k
                const bool h16 = lane & 16, h8 = lane & 8;
                double cj, ck;
                {
                    R p0 = sel(h16, fj[2], fj[0]) + __shfl_xor_sync(kAll, sel(h16, fj[0], fj[2]), 16);
                    R p1 = sel(h16, fj[3], fj[1]) + __shfl_xor_sync(kAll, sel(h16, fj[1], fj[3]), 16);
                    cj = double(sel(h8, p1, p0) + __shfl_xor_sync(kAll, sel(h8, p0, p1), 8));
                    p0 = sel(h16, fk[2], fk[0]) + __shfl_xor_sync(kAll, sel(h16, fk[0], fk[2]), 16);
                    p1 = sel(h16, fk[3], fk[1]) + __shfl_xor_sync(kAll, sel(h16, fk[1], fk[3]), 16);
                    ck = double(sel(h8, p1, p0) + __shfl_xor_sync(kAll, sel(h8, p0, p1), 8));
                }
                if (aj >= 0) fixed_add(fxf + (size_t)8 * aj + 2 * q, cj, fe);
                if (ak >= 0) fixed_add(fxf + (size_t)8 * ak + 2 * q, ck, fxe + (size_t)kTileSums * (id.t8 + K));
                if (PER) {
                    // sum of F (x) T over the images: the roots' and k's
                    double kc = ck;
                    for (int o = 4; o > 0; o >>= 1) kc += __shfl_xor_sync(kAll, kc, o);
                    for (int d = 0; d < 3; d++)
                        for (int o = 8; o <= 16; o <<= 1) vr[d] += __shfl_xor_sync(kAll, vr[d], o);
                    // lane 2c of quarter 0 holds the roots' component c; quarter c holds k's
                    const int comp = lane >> 1;
                    const double kcc = __shfl_sync(kAll, kc, (8 * comp) & 31);
                    if (lane < 6 && !(lane & 1)) {
                        fixed_add(fe + 2 * (1 + 3 * comp), ::fma(kcc, kx, vr[0]), fe);
                        fixed_add(fe + 2 * (2 + 3 * comp), ::fma(kcc, ky, vr[1]), fe);
                        fixed_add(fe + 2 * (3 + 3 * comp), ::fma(kcc, kz, vr[2]), fe);
                    }
                }
            }
            __syncwarp();
        }
    }
}

// Accumulators into the FP64 arrays, one thread per tile slot: gradient and
// dE/dCN, and per atom the three-body energy and virial (the tile's first slot
// takes the tile's energy and image terms).  The virial of all triples is
// sum F_a (x) x_a over the atoms, at their images, the origin being free.
__global__ void k_atm_finish(Batch b, Config c, AtmView v, int ntiles8, double s9, const unsigned long long* fxf,
                             const unsigned long long* fxe, const unsigned long long* queue, const int* guard, Work w,
                             double* e3, double* sig3)
{
    pdl_wait();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= kT8 * ntiles8 || (guard && *guard)) return;
    if (slot == 0 && w.counts) w.counts[1] += queue[1] / 3;
    const int a = v.sub[slot];
    if (a < 0) return;
    const bool first = (slot & 7) == 0;
    const unsigned long long* fe = fxe + (size_t)kTileSums * (slot >> 3);
    // NaN for a marked tile (and for an atom without a position, whose tile may be out of reach)
    const double nan = fe[kTileMark] || !isfinite(b.x[a] + b.y[a] + b.z[a]) ? CUDART_NAN : 0.0;
    e3[a] = (first ? s9 * fixed_value(fe) : 0.0) + nan;
    if (!c.grad) return;
    const unsigned long long* f = fxf + (size_t)8 * a;
    const double g[3] = {2.0 * s9 * fixed_value(f) + nan, 2.0 * s9 * fixed_value(f + 2) + nan,
                         2.0 * s9 * fixed_value(f + 4) + nan};
    for (int k = 0; k < 3; k++) w.grad[3 * a + k] += g[k];
    w.dEdcn[a] += s9 * fixed_value(f + 6) + nan;
    const int o = b.atom_off[b.sys_of_atom[a]];
    const double x = b.x[a] - b.x[o], y = b.y[a] - b.y[o], z = b.z[a] - b.z[o];
    double s[kSigma] = {g[0] * x, g[1] * y, g[2] * z, 0.5 * (g[0] * y + g[1] * x), 0.5 * (g[0] * z + g[2] * x),
                        0.5 * (g[1] * z + g[2] * y)};
    if (first) {
        double t[9];
        for (int k = 0; k < 9; k++) t[k] = 2.0 * s9 * fixed_value(fe + 2 * (1 + k));
        s[0] += t[0]; s[1] += t[4]; s[2] += t[8];
        s[3] += 0.5 * (t[1] + t[3]); s[4] += 0.5 * (t[2] + t[6]); s[5] += 0.5 * (t[5] + t[7]);
    }
    for (int k = 0; k < kSigma; k++) sig3[kSigma * a + k] = s[k];
}

template <class R, bool GRAD, bool PER, bool GEN>
int atm_configure()
{
    // an error here stays the last one, which the engine checks after its launches
    static PerDevice<int> blocks;
    int device = 0;
    cudaGetDevice(&device);
    const auto kernel = k_atm_triples<R, GRAD, PER, GEN>;
    const int n = blocks.get(device, (const void*)kernel, [&](int& n) {
        const int smem = (int)sizeof(AtmShared<R>) * kAtmWarps;
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
               cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 32 * kAtmWarps, smem) == cudaSuccess && n > 0;
    });
    return n > 0 ? n : 1;
}

template <class R, bool GRAD, bool PER>
int atm_occupancy_of(bool gen) { return gen ? atm_configure<R, GRAD, PER, true>() : atm_configure<R, GRAD, PER, false>(); }

template <class R, bool GRAD, bool PER, bool GEN>
void triples_t(const AtmLaunch& l)
{
    atm_configure<R, GRAD, PER, GEN>();
    launch_pdl(k_atm_triples<R, GRAD, PER, GEN>, dim3(l.blocks), dim3(32 * kAtmWarps),
               sizeof(AtmShared<R>) * kAtmWarps, l.stream, l.b, l.c, l.part, l.v, l.alp3, l.split, l.grab, l.queue,
               l.fxf, l.fxe, l.counting ? 1 : 0, l.guard);
}

template <class R, bool GRAD>
void triples_g(const AtmLaunch& l)
{
    const bool gen = l.part.nparts > 1 || l.counting;
    if (l.periodic) { if (gen) triples_t<R, GRAD, true, true>(l); else triples_t<R, GRAD, true, false>(l); }
    else { if (gen) triples_t<R, GRAD, false, true>(l); else triples_t<R, GRAD, false, false>(l); }
}

}  // namespace

size_t atm_block_bytes(bool mixed, bool grad)
{
    return kRecs * ((mixed ? sizeof(float4) : sizeof(double4)) + (grad ? (mixed ? sizeof(float2) : sizeof(double2)) : 0));
}

size_t atm_rec_bytes(bool mixed) { return kRecs * (mixed ? sizeof(float4) : sizeof(double4)); }

int atm_warps_per_block() { return kAtmWarps; }

int atm_blocks_per_sm(bool mixed, bool grad, bool periodic, bool gen)
{
    if (mixed) {
        if (grad) return periodic ? atm_occupancy_of<float, true, true>(gen) : atm_occupancy_of<float, true, false>(gen);
        return periodic ? atm_occupancy_of<float, false, true>(gen) : atm_occupancy_of<float, false, false>(gen);
    }
    if (grad) return periodic ? atm_occupancy_of<double, true, true>(gen) : atm_occupancy_of<double, true, false>(gen);
    return periodic ? atm_occupancy_of<double, false, true>(gen) : atm_occupancy_of<double, false, false>(gen);
}

size_t atm_scan_temp_bytes(long long n)
{
    size_t bytes = 0;
    const cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const int*)nullptr, (int*)nullptr, n + 1);
    return e == cudaSuccess ? bytes : 0;
}

void launch_atm_order(const Batch& b, const int* tile_off, const int* tile_sys, int ntiles, const AtmView& v,
                      double4* spheres, unsigned long long* fxf, unsigned long long* fxe, unsigned long long* queue,
                      cudaStream_t stream)
{
    if (ntiles <= 0) return;
    launch_pdl(k_atm_order, dim3((ntiles + 3) / 4), dim3(128), 0, stream, b, tile_off, tile_sys, ntiles, v, spheres, fxf,
               fxe, queue);
}

cudaError_t launch_atm_mark(const Batch& b, const Config& c, const AtmView& v, const double4* spheres, int* flag, int* map,
                            void* temp, size_t temp_bytes, cudaStream_t stream)
{
    const cudaError_t e = cudaMemsetAsync(flag + v.ncand, 0, sizeof(int), stream);
    if (e != cudaSuccess) return e;
    k_atm_mark<<<(unsigned)((v.ncand + 127) / 128), 128, 0, stream>>>(b, c, v, spheres, flag);
    return cub::DeviceScan::ExclusiveSum(temp, temp_bytes, flag, map, v.ncand + 1, stream);
}

void launch_atm_guard(const int* total, long long cap, int* guard, bool first, cudaStream_t stream)
{
    k_atm_guard<<<1, 1, 0, stream>>>(total, cap, guard, first);
}

void launch_atm_pairs(const Batch& b, const Species& s, const Config& c, const Work& w, const AtmView& v, const void* U,
                      double alp3, const int* guard, cudaStream_t stream)
{
    if (v.ncand <= 0) return;
    const unsigned blocks = (unsigned)((v.ncand + 7) / 8);
    if (c.mixed) launch_pdl(k_atm_pairs<float>, dim3(blocks), dim3(256), 0, stream, b, s, c, w, v, (const float*)U, alp3, guard);
    else launch_pdl(k_atm_pairs<double>, dim3(blocks), dim3(256), 0, stream, b, s, c, w, v, (const double*)U, alp3, guard);
}

void launch_atm_lists(const AtmView& v, int ntiles8, const int* tile8_sys, const int* sys_group, int group,
                      const long long* list_off, int4* list, int2* range, const int* guard, cudaStream_t stream)
{
    if (ntiles8 <= 0) return;
    launch_pdl(k_atm_lists, dim3((ntiles8 + 3) / 4), dim3(128), 0, stream, v, ntiles8, tile8_sys, sys_group, group,
               list_off, list, range, guard);
}

void launch_atm_triples(const AtmLaunch& l)
{
    if (l.v.ncand <= 0) return;
    if (l.c.mixed) { if (l.c.grad) triples_g<float, true>(l); else triples_g<float, false>(l); }
    else { if (l.c.grad) triples_g<double, true>(l); else triples_g<double, false>(l); }
}

void launch_atm_finish(const Batch& b, const Config& c, const AtmView& v, int ntiles8, double s9,
                       const unsigned long long* fxf, const unsigned long long* fxe, const unsigned long long* queue,
                       const int* guard, const Work& w, double* e3, double* sig3, cudaStream_t stream)
{
    if (ntiles8 <= 0) return;
    launch_pdl(k_atm_finish, dim3((kT8 * ntiles8 + 127) / 128), dim3(128), 0, stream, b, c, v, ntiles8, s9, fxf, fxe,
               queue, guard, w, e3, sig3);
}

}  // namespace d3
