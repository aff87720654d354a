// Small molecules (one lattice point, at most kMolAtoms atoms) in one or two
// kernels, one thread-block cluster per system, one warp per atom.
//
//   k_mol_pairs   coordination numbers, reference weights and species vectors,
//                 two-body sum, and without the three-body term the CN chain rule and
//                 the results; with it, the atom arrays and cleared accumulators of
//                 the three-body kernels (d3_atm.cu)
//   k_mol_finish  after the three-body kernels: their sums, the chain rule, the results
//
// What bounds it: latency.  The phases of a 12-atom molecule take a microsecond or
// two each, a kernel boundary about as much and a copy to or from the device more, so
// the phases meet at cluster barriers instead of kernel ends, positions and dE/dCN are
// exchanged through distributed shared memory, the lane keeps the CN derivative of
// its pairs in registers from the first phase to the last, and the kernel reads the
// positions from and writes the results to pinned host memory where the call has host
// buffers.  Four staged kernels and two copies before, one or (with the three-body
// term) four launches now, a call of the C entry: 12 atoms 33 -> 21 us, 100 atoms 34
// -> 27 us and with the three-body term 68 -> 50 us, 251 atoms (zero damping) 38 -> 35
// us (16 SMs share the FP64 work of 63 000 pair ends then: 25 us in the kernel).  Up to
// a microsecond of it is the barrier before the first remote store.
#include <cooperative_groups.h>
#include <math_constants.h>

#include <cfloat>
#include <cstdint>

#include "d3_atm_common.cuh"
#include "d3_damping.cuh"
#include "d3_device.cuh"
#include "d3_math.cuh"
#include "d3_per_device.h"
#include "d3_weights.cuh"

namespace d3 {

namespace {

namespace cg = cooperative_groups;

constexpr int kMolWarps = 16;                        // atoms per block
constexpr int kMolThreads = 32 * kMolWarps;
constexpr int kMolCluster = kMolAtoms / kMolWarps;   // blocks of the largest system
constexpr int kMolSteps = kMolAtoms / 32;            // partners of a lane
constexpr double kKcnMol = 16.0;                     // ncoord.f90:31
static_assert(kMolCluster <= 16, "cluster size");

// The two halves of a cluster barrier.  A block's shared memory may be touched by the
// others only once the block has started, which nothing but a barrier of the cluster
// tells: a kernel arrives at its entry and waits before its first remote store.
__device__ __forceinline__ void mol_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void mol_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ double mol_wsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Dynamic part of k_mol_pairs: the reference weights of every atom, and of every
// warp's atom i the sums V[s][q] = sum_r gw_i[r] C6ref(r of s_i, q of s) and dV with
// dgw_i: C6_ij and dC6_ij/dCN_i are seven-term products with the partner's weights.
template <class R>
__host__ __device__ constexpr size_t mol_dynamic_bytes(int nid)
{
    return sizeof(R) * ((size_t)kMolAtoms * kMaxRef + (size_t)kMolWarps * nid * 2 * kMaxRef);
}

struct MolShared {
    double pos[3 * kMolAtoms];
    double de[kMolAtoms];             // dE/dCN of every atom
    int sp[kMolAtoms];
    double wred[kMolWarps][7];        // energy and virial of the block's atoms
    double cred[kMolCluster][7];      // of the cluster's blocks (rank 0)
};

// Energy and virial of the system: the warps' sums in warp order, then the blocks' in
// rank order; v: the atom's values in all lanes (zero without an atom).
template <bool GRAD>
__device__ __forceinline__ void mol_reduce(cg::cluster_group& cluster, MolShared& sh, double (&v)[7], int rank,
                                           int nranks, int wid, int lane, int sys, double* energies, double* sigma9)
{
    constexpr int NV = GRAD ? 7 : 1;
    if (lane == 0)
        for (int k = 0; k < NV; k++) sh.wred[wid][k] = v[k];
    __syncthreads();
    if (wid == 0 && lane < NV) {
        double t = 0.0;
        for (int q = 0; q < kMolWarps; q++) t += sh.wred[q][lane];
        cluster.map_shared_rank(&sh.cred[rank][lane], 0)[0] = t;
    }
    cluster.sync();
    if (rank != 0 || wid != 0 || lane >= NV) return;
    double t = 0.0;
    for (int q = 0; q < nranks; q++) t += sh.cred[q][lane];
    if (lane == 0) {
        if (energies) energies[sys] = t;
    } else if (sigma9) {
        // Fortran sigma(3,3): element (a, b) at a + 3 b; packed xx yy zz xy xz yz
        constexpr int kAt[kSigma][2] = {{0, 0}, {4, 4}, {8, 8}, {1, 3}, {2, 6}, {5, 7}};
        sigma9[9 * sys + kAt[lane - 1][0]] = t;
        sigma9[9 * sys + kAt[lane - 1][1]] = t;
    }
}

// CN chain rule of atom i over the lane's partners (add_coordination_number_derivs,
// ncoord.f90:152-228): gradient and half the virial of every pair from both ends.
template <class R>
__device__ __forceinline__ void mol_chain(const MolShared& sh, const R (&fk)[kMolSteps], int n, int i, int lane,
                                          double& gx, double& gy, double& gz, double (&s)[kSigma])
{
    const double xi = sh.pos[3 * i], yi = sh.pos[3 * i + 1], zi = sh.pos[3 * i + 2], di = sh.de[i];
#pragma unroll
    for (int k = 0; k < kMolSteps; k++) {
        const int j = lane + 32 * k;
        if (32 * k >= n) break;
        if (j >= n || fk[k] == R(0)) continue;
        const R vx = R(xi - sh.pos[3 * j]), vy = R(yi - sh.pos[3 * j + 1]), vz = R(zi - sh.pos[3 * j + 2]);
        const R f = fk[k] * R(di + sh.de[j]);
        const R cx = f * vx, cy = f * vy, cz = f * vz;
        gx += double(cx); gy += double(cy); gz += double(cz);
        s[0] += double(R(0.5) * cx * vx); s[1] += double(R(0.5) * cy * vy); s[2] += double(R(0.5) * cz * vz);
        s[3] += double(R(0.5) * cx * vy); s[4] += double(R(0.5) * cx * vz); s[5] += double(R(0.5) * cy * vz);
    }
}

template <class R, int DAMP, bool GRAD, bool LAST>
__global__ void __launch_bounds__(kMolThreads, 1) k_mol_pairs(MolArgs a)
{
    mol_cluster_arrive();
    pdl_wait();
    __shared__ MolShared sh;
    extern __shared__ __align__(16) unsigned char smem[];
    R* sgw = reinterpret_cast<R*>(smem);                                  // [kMolAtoms][kMaxRef]
    cg::cluster_group cluster = cg::this_cluster();
    const int nranks = cluster.num_blocks(), rank = cluster.block_rank();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tid = threadIdx.x;
    const int sys = blockIdx.x / nranks;
    const Batch& b = a.b;
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    R* sv = sgw + kMolAtoms * kMaxRef + (size_t)wid * b.nid * 2 * kMaxRef;   // [nid][V 7, dV 7]
    // the block's atoms to every block of the cluster
    const int kpos = 3 * kMolWarps * rank + tid;
    const bool has_pos = tid < 3 * kMolWarps && kpos < 3 * n;
    const double vpos = has_pos ? a.pos[3 * (size_t)a0 + kpos] : 0.0;
    for (int k = tid; k < n; k += kMolThreads) sh.sp[k] = b.sp[a0 + k];
    mol_cluster_wait();
    if (has_pos)
        for (int r = 0; r < nranks; r++) cluster.map_shared_rank(&sh.pos[kpos], r)[0] = vpos;
    cluster.sync();

    const int i = kMolWarps * rank + wid;
    const bool active = i < n;
    const int ic = active ? i : 0;
    const double xi = sh.pos[3 * ic], yi = sh.pos[3 * ic + 1], zi = sh.pos[3 * ic + 2];
    const int si = sh.sp[ic], nid = b.nid;
    R fk[kMolSteps];                       // CN derivative of the lane's pairs: dcf / r
    // ---- coordination number (ncoord.f90:86-144) and weights
    if (active) {
        const double rci = a.s.rcov[si];
        const R cut2 = R(a.c.cut_cn * a.c.cut_cn);
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < kMolSteps; k++) {
            fk[k] = R(0);
            const int j = lane + 32 * k;
            if (32 * k >= n) break;
            if (j >= n) continue;
            const R vx = R(xi - sh.pos[3 * j]), vy = R(yi - sh.pos[3 * j + 1]), vz = R(zi - sh.pos[3 * j + 2]);
            const R r2 = vx * vx + vy * vy + vz * vz;
            if (r2 > cut2 || r2 < R(1.0e-12)) continue;
            const R rc = R(rci + a.s.rcov[sh.sp[j]]);
            R ir, cf;
            if constexpr (sizeof(R) == 8) {
                ir = rsqrt_fast(r2);
                cf = rcp_fast(R(1) + exp(-R(kKcnMol) * (rc * ir - R(1))));
            } else {
                ir = rsqrtf(r2);
                cf = R(1) / (R(1) + expf(-R(kKcnMol) * (rc * ir - R(1))));
            }
            acc += double(cf);
            if (GRAD) fk[k] = -cf * (R(1) - cf) * R(kKcnMol) * rc * (ir * ir * ir);
        }
        acc = mol_wsum(acc);
        if (lane == 0) a.w.cn[a0 + i] = acc;
        // the three-body kernels read the species vectors, the two-body sum below V
        atom_weights<R>(b, a.s, a.c, a.w, a0 + i, acc, lane, LAST ? (R*)nullptr : (R*)a.UV);
        __syncwarp();
        double g[kMaxRef], dg[kMaxRef];
#pragma unroll
        for (int r = 0; r < kMaxRef; r++) {
            g[r] = a.w.gw[(size_t)(a0 + i) * kMaxRef + r];
            dg[r] = a.w.dgw[(size_t)(a0 + i) * kMaxRef + r];
        }
        if (lane < nranks) {
            // a ghost's weights are zero here: no C6 with it
            const bool ghost = b.ghost && b.ghost[a0 + i];
            R* to = cluster.map_shared_rank(sgw + i * kMaxRef, lane);
#pragma unroll
            for (int r = 0; r < kMaxRef; r++) to[r] = ghost ? R(0) : R(g[r]);
        }
        const double* ref = a.s.c6ref + (size_t)si * nid * kMaxRef * kMaxRef;
        for (int e = lane; e < nid * kMaxRef; e += 32) {
            const int s_ = e / kMaxRef, q = e % kMaxRef;
            double v = 0.0, dv = 0.0;
#pragma unroll
            for (int r = 0; r < kMaxRef; r++) {
                const double c6 = __ldg(ref + ((size_t)s_ * kMaxRef + r) * kMaxRef + q);
                v += g[r] * c6;
                dv += dg[r] * c6;
            }
            sv[s_ * 2 * kMaxRef + q] = R(v);
            sv[s_ * 2 * kMaxRef + kMaxRef + q] = R(dv);
        }
    }
    cluster.sync();

    // ---- two-body sum (rational.f90:378-514, zero.f90:409-553 and the other families)
    double e = 0.0, de = 0.0, gx = 0.0, gy = 0.0, gz = 0.0, sg[kSigma] = {0, 0, 0, 0, 0, 0};
    if (active && a.two_body && !(b.ghost && b.ghost[a0 + i])) {
        const R cutoff = R(a.c.cut2), cut2 = R(a.c.cut2 * a.c.cut2), width = R(a.c.width2);
        const bool smooth = a.c.width2 > 0.0 && a.c.width2 < a.c.cut2;
        const R s6 = R(a.d.s6), s8 = R(a.d.s8), alp6 = R(a.d.alp), alp8 = R(a.d.alp + 2.0), bet = R(a.d.bet),
                a1 = R(a.d.a1);
        const int h6 = half_even(a.d.alp), hb = half_even(a.d.bet);
        const int zi_ = DAMP == kZDamping ? b.zid[a0 + i] : 0;
        for (int j = lane; j < n; j += 32) {
            const R vx = R(xi - sh.pos[3 * j]), vy = R(yi - sh.pos[3 * j + 1]), vz = R(zi - sh.pos[3 * j + 2]);
            const R r2 = vx * vx + vy * vy + vz * vz;
            if (r2 > cut2 || r2 < R(DBL_EPSILON)) continue;
            const int sj = sh.sp[j];
            R c6 = R(0), dc6i = R(0);
#pragma unroll
            for (int q = 0; q < kMaxRef; q++) {
                const R gj = sgw[j * kMaxRef + q];
                c6 += sv[sj * 2 * kMaxRef + q] * gj;
                dc6i += sv[sj * 2 * kMaxRef + kMaxRef + q] * gj;
            }
            if (c6 == R(0)) continue;
            const double2* pr = reinterpret_cast<const double2*>(a.s.pair + kPairSlots * (si * nid + sj));
            const double2 p01 = __ldg(pr), p23 = __ldg(pr + 1), p45 = __ldg(pr + 2);
            const R rrij = R(p01.x), q1 = R(p01.y), q2 = R(p23.x), q3 = R(p23.y), q4 = R(p45.x), q5 = R(p45.y);
            R sw = R(1), dsw = R(0), r1 = R(1);
            if (smooth) {
                r1 = tt_sqrt<R>(r2);
                tt_smooth<R>(r1, cutoff, width, sw, dsw);
            }
            R ed, gd, cd = R(0);
            if constexpr (DAMP == kRational) {
                const R r4 = r2 * r2;
                const R a6 = r4 * r2 + q1, a8 = r4 * r4 + q2;
                const R ia = inv<R>(a6 * a8);
                const R t6 = a8 * ia, t8 = a6 * ia;
                const R s8rr = s8 * rrij;
                ed = s6 * t6 + s8rr * t8;
                gd = r4 * (R(-6) * s6 * t6 * t6 + R(-8) * s8rr * r2 * t8 * t8);
            } else if constexpr (DAMP == kZero) {
                const R ir2 = inv<R>(r2);
                const R ir6 = ir2 * ir2 * ir2;
                R t6, t8;
                if (h6 >= 0) {
                    t6 = ipow(q1 * q1 * ir2, h6);
                    t8 = ipow(q2 * q2 * ir2, h6 + 1);
                } else {
                    if (!smooth) r1 = tt_sqrt<R>(r2);
                    t6 = tt_pow<R>(q1 / r1, alp6);
                    t8 = tt_pow<R>(q2 / r1, alp8);
                }
                t6 = damping_power(t6); t8 = damping_power(t8);
                const R f6 = inv<R>(R(1) + R(6) * t6), f8 = inv<R>(R(1) + R(6) * t8);
                const R w6 = s6 * ir6, w8 = s8 * rrij * (ir6 * ir2);
                ed = w6 * f6 + w8 * f8;
                gd = ir2 * (w6 * f6 * (R(-6) + R(6) * alp6 * t6 * f6) + w8 * f8 * (R(-8) + R(6) * alp8 * t8 * f8));
            } else {
                const R zc = DAMP == kZDamping ? a1 / R(zi_ + b.zid[a0 + j]) * c6 : R(0);
                tt_family<R, DAMP>(r2, r1, smooth, rrij, q1, q2, q3, q4, q5, zc, s6, s8, alp6, alp8, bet, a1, h6, hb, ed,
                                   gd, cd);
            }
            // E = -C6 ed / 2 per end, dE/dCN = -dC6/dCN ed, gradient -C6 gd v
            const R edisp = sw * ed;
            e += double(R(-0.5) * c6 * edisp);
            if (!GRAD) continue;
            de -= double(dc6i * (DAMP == kZDamping ? sw * cd : edisp));
            R gdisp = sw * gd;
            if (smooth) gdisp += dsw * ed / r1;
            const R f = -c6 * gdisp;
            const R cx = f * vx, cy = f * vy, cz = f * vz;
            gx += double(cx); gy += double(cy); gz += double(cz);
            sg[0] += double(R(0.5) * cx * vx); sg[1] += double(R(0.5) * cy * vy); sg[2] += double(R(0.5) * cz * vz);
            sg[3] += double(R(0.5) * cx * vy); sg[4] += double(R(0.5) * cx * vz); sg[5] += double(R(0.5) * cy * vz);
        }
    }
    if (LAST && GRAD) {
        de = mol_wsum(de);
        if (active && lane < nranks) cluster.map_shared_rank(&sh.de[i], lane)[0] = de;
        cluster.sync();
        if (active) mol_chain<R>(sh, fk, n, i, lane, gx, gy, gz, sg);
    }
    e = mol_wsum(e);
    if (GRAD) {
        gx = mol_wsum(gx); gy = mol_wsum(gy); gz = mol_wsum(gz);
        for (int k = 0; k < kSigma; k++) sg[k] = mol_wsum(sg[k]);
    }
    if (LAST) {
        if (GRAD && active && a.grad_out && lane < 3)
            a.grad_out[3 * (size_t)(a0 + i) + lane] = lane == 0 ? gx : lane == 1 ? gy : gz;
        double v[7] = {e, sg[0], sg[1], sg[2], sg[3], sg[4], sg[5]};
        mol_reduce<GRAD>(cluster, sh, v, rank, nranks, wid, lane, sys, a.energies, a.sigma9);
    } else {
        // for the three-body kernels and k_mol_finish
        if (GRAD) de = mol_wsum(de);
        const int slot = kMolSlots * a.v.t8_off[sys] + i;
        if (i < kMolSlots * ((n + kMolSlots - 1) / kMolSlots)) {
            if (lane == 0) {
                a.v.sub[slot] = active ? a0 + i : -1;
                a.v.pos[slot] = active ? make_double4(xi, yi, zi, (double)(a0 + i)) : make_double4(0.0, 0.0, 0.0, 0.0);
            }
            if (i % kMolSlots == 0 && lane < kTileSums) a.fxe[(size_t)kTileSums * (slot / kMolSlots) + lane] = 0;
        }
        if (sys == 0 && rank == 0 && tid < 2) a.queue[tid] = 0;
        if (active) {
            if (GRAD && lane < 8) a.fxf[(size_t)8 * (a0 + i) + lane] = 0;
            if (lane == 0) {
                a.x[a0 + i] = xi; a.y[a0 + i] = yi; a.z[a0 + i] = zi;
                a.w.e_atom[a0 + i] = e;
                if (GRAD) {
                    a.w.dEdcn[a0 + i] = de;
                    a.w.grad[3 * (a0 + i)] = gx; a.w.grad[3 * (a0 + i) + 1] = gy; a.w.grad[3 * (a0 + i) + 2] = gz;
                    for (int k = 0; k < kSigma; k++) a.w.sig_atom[kSigma * (a0 + i) + k] = sg[k];
                }
            }
            if (GRAD) {
                R* fs = (R*)a.fstore + (size_t)(a0 + i) * kMolAtoms;
#pragma unroll
                for (int k = 0; k < kMolSteps; k++)
                    if (lane + 32 * k < n) fs[lane + 32 * k] = fk[k];
            }
        }
    }
}

// Adds the three-body sums (fixed point) to the two-body results, then the CN chain
// rule with the complete dE/dCN, and the per-system results.
template <class R, bool GRAD>
__global__ void __launch_bounds__(kMolThreads, 1) k_mol_finish(MolArgs a)
{
    pdl_wait();
    __shared__ MolShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    const int nranks = cluster.num_blocks(), rank = cluster.block_rank();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tid = threadIdx.x;
    const int sys = blockIdx.x / nranks;
    const Batch& b = a.b;
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    const double s9 = a.d.s9;
    // NaN for a marked tile
    const unsigned long long* fe = a.fxe + (size_t)kTileSums * a.v.t8_off[sys];
    auto mark = [&](int k) { return fe[(size_t)kTileSums * (k / kMolSlots) + kTileMark] ? CUDART_NAN : 0.0; };
    if (GRAD)
        for (int k = tid; k < n; k += kMolThreads) {
            sh.pos[3 * k] = a.x[a0 + k]; sh.pos[3 * k + 1] = a.y[a0 + k]; sh.pos[3 * k + 2] = a.z[a0 + k];
            sh.de[k] = a.w.dEdcn[a0 + k] + s9 * fixed_value(a.fxf + (size_t)8 * (a0 + k) + 6) + mark(k);
        }
    cluster.sync();
    const int i = kMolWarps * rank + wid;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    if (i < n) {
        const double nan = mark(i);
        v[0] = a.w.e_atom[a0 + i] + nan;
        if (i % kMolSlots == 0) v[0] += s9 * fixed_value(fe + (size_t)kTileSums * (i / kMolSlots));
        if (GRAD) {
            R fk[kMolSteps];
            const R* fs = (const R*)a.fstore + (size_t)(a0 + i) * kMolAtoms;
#pragma unroll
            for (int k = 0; k < kMolSteps; k++) fk[k] = lane + 32 * k < n ? fs[lane + 32 * k] : R(0);
            double gx = 0, gy = 0, gz = 0, sg[kSigma] = {0, 0, 0, 0, 0, 0};
            mol_chain<R>(sh, fk, n, i, lane, gx, gy, gz, sg);
            gx = mol_wsum(gx); gy = mol_wsum(gy); gz = mol_wsum(gz);
            for (int k = 0; k < kSigma; k++) sg[k] = mol_wsum(sg[k]);
            const unsigned long long* f = a.fxf + (size_t)8 * (a0 + i);
            const double tx = 2.0 * s9 * fixed_value(f) + nan, ty = 2.0 * s9 * fixed_value(f + 2) + nan,
                         tz = 2.0 * s9 * fixed_value(f + 4) + nan;
            // the three-body virial is sum F_a (x) x_a, the origin being free
            const double x = sh.pos[3 * i] - sh.pos[0], y = sh.pos[3 * i + 1] - sh.pos[1], z = sh.pos[3 * i + 2] - sh.pos[2];
            const double t3[kSigma] = {tx * x, ty * y, tz * z, 0.5 * (tx * y + ty * x), 0.5 * (tx * z + tz * x),
                                       0.5 * (ty * z + tz * y)};
            const double* g2 = a.w.grad + 3 * (size_t)(a0 + i);
            if (a.grad_out && lane < 3)
                a.grad_out[3 * (size_t)(a0 + i) + lane] = (lane == 0 ? gx + tx : lane == 1 ? gy + ty : gz + tz) + g2[lane];
            for (int k = 0; k < kSigma; k++) v[1 + k] = a.w.sig_atom[kSigma * (a0 + i) + k] + sg[k] + t3[k];
        }
    }
    mol_reduce<GRAD>(cluster, sh, v, rank, nranks, wid, lane, sys, a.energies, a.sigma9);
}

using MolKernel = void (*)(MolArgs);

// Clusters above eight blocks need a kernel's consent, given once on each device.
bool mol_consent(MolKernel kernel)
{
    static PerDevice<bool> consent;
    int device = 0;
    cudaGetDevice(&device);
    return consent.get(device, (const void*)kernel, [&](bool& ok) {
        ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        return ok;
    });
}

void mol_launch(MolKernel kernel, const MolArgs& a, int cluster, size_t smem, cudaStream_t stream)
{
    // without consent the launch fails, and the engine reports its error
    if (cluster > 8) mol_consent(kernel);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.b.nsys * cluster);
    cfg.blockDim = dim3(kMolThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kernel, a);
}

template <class R, int DAMP>
MolKernel mol_pairs_kernel(bool grad, bool last)
{
    if (grad) return last ? k_mol_pairs<R, DAMP, true, true> : k_mol_pairs<R, DAMP, true, false>;
    return last ? k_mol_pairs<R, DAMP, false, true> : k_mol_pairs<R, DAMP, false, false>;
}

template <class R>
MolKernel mol_pairs_kernel(int kind, bool grad, bool last)
{
    switch (kind) {
    case kRational: return mol_pairs_kernel<R, kRational>(grad, last);
    case kZero: return mol_pairs_kernel<R, kZero>(grad, last);
    case kMZero: return mol_pairs_kernel<R, kMZero>(grad, last);
    case kOptimizedPower: return mol_pairs_kernel<R, kOptimizedPower>(grad, last);
    case kCSO: return mol_pairs_kernel<R, kCSO>(grad, last);
    default: return mol_pairs_kernel<R, kZDamping>(grad, last);
    }
}

}  // namespace

int mol_cluster_size(int max_atoms)
{
    int c = 1;
    while (c * kMolWarps < max_atoms) c *= 2;
    return c;
}

bool mol_cluster_fits(int cluster)
{
    if (cluster <= 8) return true;
    static PerDevice<bool> fits;
    int device = 0;
    cudaGetDevice(&device);
    const MolKernel kernel = k_mol_pairs<double, kRational, true, true>;
    const bool ok = fits.get(device, (const void*)kernel, [&](bool& ok) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMolCluster);
        cfg.blockDim = dim3(kMolThreads);
        cfg.dynamicSmemBytes = mol_dynamic_bytes<double>(kMolSpecies);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kMolCluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        ok = mol_consent(kernel) && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
        return ok;
    });
    if (!ok) (void)cudaGetLastError();        // the staged kernels serve these systems
    return ok;
}

void launch_mol_pairs(const MolArgs& a, int cluster, bool last, cudaStream_t stream)
{
    mol_launch(a.c.mixed ? mol_pairs_kernel<float>(a.d.kind, a.c.grad, last)
                         : mol_pairs_kernel<double>(a.d.kind, a.c.grad, last), a, cluster,
               a.c.mixed ? mol_dynamic_bytes<float>(a.b.nid) : mol_dynamic_bytes<double>(a.b.nid), stream);
}

void launch_mol_finish(const MolArgs& a, int cluster, cudaStream_t stream)
{
    if (a.c.mixed) mol_launch(a.c.grad ? k_mol_finish<float, true> : k_mol_finish<float, false>, a, cluster, 0, stream);
    else mol_launch(a.c.grad ? k_mol_finish<double, true> : k_mol_finish<double, false>, a, cluster, 0, stream);
}

}  // namespace d3
