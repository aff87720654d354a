// Pairwise decomposition of the dispersion energy (get_pairwise_dispersion_v2,
// disp.f90:403-457), in FP64: the additive (two-body) energy of every atom
// pair and the non-additive (ATM) energy distributed over the pairs of each
// triple, as the matrices energy2[i][j] and energy3[i][j] of every system
// (input atom order, systems one after the other).
//
//   k_pw_c6        C6 of every ordered atom pair of each system (sorted order), and for
//                  systems of one lattice point the pair's factors {m, P} of a triple
//   k_pw_factors   these factors of every ordered pair and translation
//   k_pw_near      the sites within the cutoff of every atom
//   k_pairwise2    one block per atom i: the lanes take the partners j and sum
//                  the pair over all lattice translations; every (i, j) entry
//                  is written once by its row, no atomics
//   k_pairwise3    one warp per atom pair (i, j <= i): the energies of all triples
//                  (atm.f90:829-950) that hold the pair, the lanes taking the third
//                  atoms and images; a sixth of each triple energy belongs to each
//                  ordered pair of the triple, so the entry is a sixth of that sum
#include <cfloat>
#include <cstdint>

#include "d3_device.cuh"
#include "d3_atm_common.cuh"

namespace d3 {

namespace {

constexpr int kPwThreads = 128;

__device__ __forceinline__ int system_of_offset(const long long* off, int nsys, long long t)
{
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (off[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Factors of one pair of a triple (d3_atm.cu): m = sqrt(C6) r^-3 times the smooth
// switch, and the pair's share P of (r0/r)^alp3, bounded so that the product of three
// stays finite.  Zero outside the cutoff.
__device__ __forceinline__ double2 pw_factor(double x, double c6, double r0, double alp3, const Config& c)
{
    if (x > c.cut3 * c.cut3 || x < DBL_EPSILON || c6 == 0.0) return make_double2(0.0, 0.0);
    const double u = 1.0 / x;
    double m = sqrt(fabs(c6)) * u * sqrt(u);
    if (c.width3 > 0.0) {
        double sw, dsw;
        smooth<double>(sqrt(x), c.cut3, c.width3, sw, dsw);
        m *= sw;
    }
    return make_double2(m, fmin(exp(0.5 * alp3 * log(r0 * r0 * u)), 1e100));
}

// C6 of the ordered pair (r, c) of each system (get_atomic_c6,
// model.f90:340-431); ghost atoms give 0.
__global__ void k_pw_c6(Batch b, Species s, Config cf, Work w, const long long* off, long long total, double alp3,
                        double* c6, double2* mp)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int sys = system_of_offset(off, b.nsys, t);
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    const long long e = t - off[sys];
    const int r = a0 + (int)(e / n), c = a0 + (int)(e % n);
    double v = 0.0;
    const int sr = b.sp[r], sc = b.sp[c];
    if (!(b.ghost && (b.ghost[r] || b.ghost[c]))) {
        const double* ref = s.c6ref + (size_t)(sr * b.nid + sc) * kMaxRef * kMaxRef;
        for (int ir = 0; ir < s.nref[sr]; ir++) {
            double a = 0.0;
            for (int jr = 0; jr < s.nref[sc]; jr++) a += w.gw[c * kMaxRef + jr] * __ldg(ref + ir * kMaxRef + jr);
            v += w.gw[r * kMaxRef + ir] * a;
        }
    }
    c6[t] = v;
    if (!mp) return;
    const double dx = b.x[r] - b.x[c], dy = b.y[r] - b.y[c], dz = b.z[r] - b.z[c];
    mp[t] = pw_factor(dx * dx + dy * dy + dz * dz, v, s.atm_r0[sr * b.nid + sc], alp3, cf);
}

// mp[foff[sys] + (r n + c) nT + T]: factors of (r, c at T).
__global__ void k_pw_factors(Batch b, Species s, Config cf, const long long* off, const long long* foff, long long total,
                             double alp3, const double* c6, double2* mp)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int sys = system_of_offset(foff, b.nsys, t);
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    const int t0 = b.img_off[kImgDisp3 * (b.nsys + 1) + sys], nT = b.img_off[kImgDisp3 * (b.nsys + 1) + sys + 1] - t0;
    const long long e = (t - foff[sys]) / nT;
    const double* T = b.img + 3 * (t0 + (t - foff[sys]) - e * nT);
    const int r = a0 + (int)(e / n), c = a0 + (int)(e % n);
    const double dx = b.x[c] + T[0] - b.x[r], dy = b.y[c] + T[1] - b.y[r], dz = b.z[c] + T[2] - b.z[r];
    mp[t] = pw_factor(dx * dx + dy * dy + dz * dz, c6[off[sys] + e], s.atm_r0[b.sp[r] * b.nid + b.sp[c]], alp3, cf);
}

// near[foff[sys] + r n nT + k], k < count[r]: the sites {c, T} within the cutoff of atom r
// with a nonzero factor, ascending.  One warp per atom.
__global__ void k_pw_near(Batch b, const long long* foff, const double2* mp, int2* near, int* count)
{
    const int lane = threadIdx.x & 31;
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= b.natoms) return;
    const int sys = b.sys_of_atom[r];
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    const int nT = b.img_off[kImgDisp3 * (b.nsys + 1) + sys + 1] - b.img_off[kImgDisp3 * (b.nsys + 1) + sys];
    const long long row = foff[sys] + (long long)(r - a0) * n * nT;
    int k = 0;
    for (int e0 = 0; e0 < n * nT; e0 += 32) {
        const int e = e0 + lane;
        const bool in = e < n * nT && mp[row + e].x != 0.0;
        const unsigned msk = __ballot_sync(0xffffffffu, in);
        if (in) near[row + k + __popc(msk & ((1u << lane) - 1u))] = make_int2(e / nT, e % nT);
        k += __popc(msk);
    }
    if (lane == 0) count[r] = k;
}

// edisp of one (i, j, T) term without the smooth cutoff: the energy
// expressions of rational.f90:623-705, zero.f90:662-755 and the pairwise
// routines of mzero, optimizedpower, cso and z.f90, with the pair constants
// of the engine's table (rrij, q1..q5) and, for Z damping, zc = R0 C6.
__device__ double pw_edisp(const Damp& d, const double* pr, double r2, double zc)
{
    const double rrij = pr[0];
    const double r4 = r2 * r2, r6 = r4 * r2, r8 = r6 * r2;
    switch (d.kind) {
    case kRational:
        return d.s6 / (r6 + pr[1]) + d.s8 * rrij / (r8 + pr[2]);
    case kZero: {
        const double r1 = sqrt(r2);
        const double t6 = pow(pr[1] / r1, d.alp), t8 = pow(pr[2] / r1, d.alp + 2.0);
        return d.s6 / (1.0 + 6.0 * t6) / r6 + d.s8 * rrij / (1.0 + 6.0 * t8) / r8;
    }
    case kMZero: {
        const double r1 = sqrt(r2);
        const double t6 = pow(r1 * pr[1] + pr[3], -d.alp), t8 = pow(r1 * pr[2] + pr[3], -(d.alp + 2.0));
        return d.s6 / (1.0 + 6.0 * t6) / r6 + d.s8 * rrij / (1.0 + 6.0 * t8) / r8;
    }
    case kOptimizedPower: {
        const double ib = pow(r2, -0.5 * d.bet);
        return d.s6 / (r6 + pr[1] * ib) + d.s8 * rrij / (r8 + pr[2] * ib);
    }
    case kCSO: {
        const double sf = 1.0 / (1.0 + exp(sqrt(r2) - pr[2]));
        return (d.s6 + d.a1 * sf) / (r6 + pr[1]);
    }
    default:
        return d.s6 / (r6 + zc) + d.s8 * rrij / (r8 + zc * rrij);
    }
}

__global__ void __launch_bounds__(kPwThreads) k_pairwise2(Batch b, Species s, Damp d, Config c, const long long* off,
                                                           const double* c6, double* e2)
{
    const int p = blockIdx.x;
    const int sys = b.sys_of_atom[p];
    const int a0 = b.atom_off[sys], a1 = b.atom_off[sys + 1], n = a1 - a0;
    const int t0 = b.img_off[kImgDisp2 * (b.nsys + 1) + sys], t1 = b.img_off[kImgDisp2 * (b.nsys + 1) + sys + 1];
    const double xp = b.x[p], yp = b.y[p], zp = b.z[p];
    const double cut2 = c.cut2 * c.cut2;
    const int sp = b.sp[p];
    const double* crow = c6 + off[sys] + (long long)(p - a0) * n;
    double* erow = e2 + off[sys] + (long long)b.local[p] * n;
    for (int q = a0 + threadIdx.x; q < a1; q += blockDim.x) {
        const double c6pq = crow[q - a0];
        double sum = 0.0;
        if (c6pq != 0.0) {
            const double* pr = s.pair + kPairSlots * (sp * b.nid + b.sp[q]);
            const double zc = d.kind == kZDamping ? d.a1 / double(b.zid[p] + b.zid[q]) * c6pq : 0.0;
            const double dx = xp - b.x[q], dy = yp - b.y[q], dz = zp - b.z[q];
            for (int t = t0; t < t1; t++) {
                const double vx = dx - b.img[3 * t], vy = dy - b.img[3 * t + 1], vz = dz - b.img[3 * t + 2];
                const double r2 = vx * vx + vy * vy + vz * vz;
                if (r2 > cut2 || r2 < DBL_EPSILON) continue;
                double sw = 1.0, dsw = 0.0;
                if (c.width2 > 0.0) smooth<double>(sqrt(r2), c.cut2, c.width2, sw, dsw);
                sum -= 0.5 * c6pq * sw * pw_edisp(d, pr, r2, zc);
            }
        }
        erow[b.local[q]] = sum;
    }
}

// Energy of a triple from its squared distances and the products of the pair factors.
__device__ __forceinline__ double pw_triple(double x, double y, double z, double m, double P)
{
    const double w = x * y * z;
    const double A = 0.375 * (x + y - z) * (x - y + z) * (y + z - x) / w;
    return m * (1.0 + A) / (1.0 + 6.0 * P);
}

// A site pair (i at 0, j at T_j) occurs once with every third site, also where sites
// are images of one atom (atm.f90:954-980 then weights the repeated visits of the
// reference's loop), so no weights are needed: a triple is visited three times, once
// per pair.  mp: the factors of every pair (and translation), near: the sites around
// every atom; with PER (a system has more than one lattice point) both may be null.
// What bounds it: FP64 issue, with PER the loads of the factors too.  With images most
// sites are out of reach.  A cell of 400 atoms: one thread per pair and each triple once
// 262 ms; from all sites, the factors computed per visit, 647 ms; from the table 385 ms;
// from the table and the sites in reach 88 ms (800 atoms: 369 ms, the last two 1447 and
// 218 ms; a molecule of 600 atoms 2.9 -> 1.2 ms without the code of the images).
template <bool PER>
__global__ void __launch_bounds__(kPwThreads) k_pairwise3(Batch b, Species s, Damp d, Config c, const long long* off,
                                                          const long long* foff, long long total, const double* c6,
                                                          const double2* mp, const int2* near, const int* count,
                                                          double* e3)
{
    const int lane = threadIdx.x & 31;
    const long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (t >= total) return;
    const int sys = system_of_offset(off, b.nsys, t);
    const int a0 = b.atom_off[sys], n = b.atom_off[sys + 1] - a0;
    const long long e = t - off[sys];
    const int pl = (int)(e / n), ql = (int)(e % n);
    if (ql > pl) return;                     // pairs (i, j <= i) only
    const int p = a0 + pl, q = a0 + ql;
    const double* cm = c6 + off[sys];
    const double c6pq = cm[(long long)pl * n + ql];
    double sum = 0.0;
    if (c6pq != 0.0) {
        const int t0 = b.img_off[kImgDisp3 * (b.nsys + 1) + sys];
        const int nT = PER ? b.img_off[kImgDisp3 * (b.nsys + 1) + sys + 1] - t0 : 1;
        const double* img = b.img + 3 * t0;
        const double cut2 = c.cut3 * c.cut3, alp3 = (d.alp + 2.0) / 3.0;
        const int sp = b.sp[p], sq = b.sp[q];
        const double xp = b.x[p], yp = b.y[p], zp = b.z[p];
        // factors of i and of j with every site
        const long long row = PER ? foff[sys] + (long long)pl * n * nT : off[sys] + (long long)pl * n;
        const double2* mpp = mp ? mp + row : nullptr;
        const double2* mpq = mp ? mp + (PER ? foff[sys] + (long long)ql * n * nT : off[sys] + (long long)ql * n) : nullptr;
        const int sites = PER && near ? count[p] : n * nT;
        for (int tj = 0; tj < nT; tj++) {
            const double tjx = PER ? img[3 * tj] : 0.0, tjy = PER ? img[3 * tj + 1] : 0.0, tjz = PER ? img[3 * tj + 2] : 0.0;
            const double ijx = b.x[q] + tjx - xp, ijy = b.y[q] + tjy - yp, ijz = b.z[q] + tjz - zp;
            const double r2ij = ijx * ijx + ijy * ijy + ijz * ijz;
            if (r2ij > cut2 || r2ij < DBL_EPSILON) continue;
            const double2 fij = !PER || mp ? mpp[(long long)ql * nT + tj]
                                           : pw_factor(r2ij, c6pq, s.atm_r0[sp * b.nid + sq], alp3, c);
            // the translations run over a box around 0 (its middle): T_k - T_j is this far on in it
            const int shift = (nT - 1) / 2 - tj;
            for (int f = lane; f < sites; f += 32) {
                int2 site = make_int2(f, 0);
                if (PER) site = near ? near[row + f] : make_int2(f / nT, f % nT);
                const int rl = site.x, tk = site.y, r = a0 + rl;
                const double tkx = PER ? img[3 * tk] : 0.0, tky = PER ? img[3 * tk + 1] : 0.0, tkz = PER ? img[3 * tk + 2] : 0.0;
                const double ikx = b.x[r] + tkx - xp, iky = b.y[r] + tky - yp, ikz = b.z[r] + tkz - zp;
                const double r2ik = ikx * ikx + iky * iky + ikz * ikz;
                if (r2ik > cut2 || r2ik < DBL_EPSILON) continue;
                const double jkx = ikx - ijx, jky = iky - ijy, jkz = ikz - ijz;
                const double r2jk = jkx * jkx + jky * jky + jkz * jkz;
                if (r2jk > cut2 || r2jk < DBL_EPSILON) continue;
                double2 fik, fjk;
                if (!PER) {
                    fik = mpp[rl];
                    fjk = mpq[rl];
                } else {
                    const int td = tk + shift;
                    if (mp) fik = mpp[(long long)rl * nT + tk];
                    else fik = pw_factor(r2ik, cm[(long long)rl * n + pl], s.atm_r0[sp * b.nid + b.sp[r]], alp3, c);
                    // from the table unless T_k - T_j lies outside the box (atoms outside the cell)
                    if (mp && (unsigned)td < (unsigned)nT &&
                        fabs(img[3 * td] - (tkx - tjx)) + fabs(img[3 * td + 1] - (tky - tjy)) +
                                fabs(img[3 * td + 2] - (tkz - tjz)) < 1e-6)
                        fjk = mpq[(long long)rl * nT + td];
                    else
                        fjk = pw_factor(r2jk, cm[(long long)rl * n + ql], s.atm_r0[sq * b.nid + b.sp[r]], alp3, c);
                }
                sum += pw_triple(r2ij, r2ik, r2jk, fij.x * fik.x * fjk.x, fij.y * fik.y * fjk.y);
            }
        }
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        sum *= d.s9 / 6.0;
    }
    if (lane != 0) return;
    double* eg = e3 + off[sys];
    const long long lp = b.local[p], lq = b.local[q];
    eg[lp * n + lq] = sum;
    eg[lq * n + lp] = sum;
}

__global__ void k_copy_out(const double* __restrict__ src, double* __restrict__ dst, long long n)
{
    pdl_wait();
    const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k < n) dst[k] = src[k];
}

}  // namespace

void launch_copy_out(const double* src, double* dst, long long n, cudaStream_t stream)
{
    if (n > 0) launch_pdl(k_copy_out, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, src, dst, n);
}

void launch_pairwise(const Batch& b, const Species& s, const Damp& d, const Config& c, const Work& w,
                     const long long* off, long long total, const long long* foff, long long ftotal, double* c6,
                     double* factors, double* e2, double* e3, cudaStream_t stream)
{
    if (b.natoms <= 0 || total <= 0) return;
    const bool threebody = std::fabs(d.s9) >= DBL_EPSILON;
    auto blocks = [](long long threads) { return (unsigned)((threads + kPwThreads - 1) / kPwThreads); };
    const double alp3 = (d.alp + 2.0) / 3.0;
    double2* mp = threebody ? reinterpret_cast<double2*>(factors) : nullptr;
    const bool molecules = ftotal == total;
    k_pw_c6<<<blocks(total), kPwThreads, 0, stream>>>(b, s, c, w, off, total, alp3, c6, molecules ? mp : nullptr);
    k_pairwise2<<<b.natoms, kPwThreads, 0, stream>>>(b, s, d, c, off, c6, e2);
    if (!threebody) {
        cudaMemsetAsync(e3, 0, sizeof(double) * total, stream);
        return;
    }
    if (molecules) {
        k_pairwise3<false><<<blocks(32 * total), kPwThreads, 0, stream>>>(b, s, d, c, off, foff, total, c6, mp, nullptr,
                                                                         nullptr, e3);
        return;
    }
    int2* near = nullptr;
    int* count = nullptr;
    if (mp) {
        near = reinterpret_cast<int2*>(mp + ftotal);
        count = reinterpret_cast<int*>(near + ftotal);
        k_pw_factors<<<blocks(ftotal), kPwThreads, 0, stream>>>(b, s, c, off, foff, ftotal, alp3, c6, mp);
        k_pw_near<<<blocks(32LL * b.natoms), kPwThreads, 0, stream>>>(b, foff, mp, near, count);
    }
    k_pairwise3<true><<<blocks(32 * total), kPwThreads, 0, stream>>>(b, s, d, c, off, foff, total, c6, mp, near, count, e3);
}

// Doubles of the factors and, with images, of the sites in reach.
size_t pairwise_factor_doubles(long long total, long long ftotal, int natoms)
{
    return ftotal == total ? 2 * (size_t)ftotal : 3 * (size_t)ftotal + ((size_t)natoms + 1) / 2;
}

}  // namespace d3
