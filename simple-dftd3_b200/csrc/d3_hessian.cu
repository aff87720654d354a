// Analytic Hessian of the dispersion energy (get_dispersion_hessian,
// disp.f90:236-308), in FP64, for one structure in input atom order.
//
//   k_hs_cn       per atom m: CN, column m of B = dCN/dR [3N][N] (ncoord.f90) and
//                 the reference weights with their first two CN derivatives
//                 (model.f90:201-273)
//   k_hs_c6       C6, dC6/dCN and the second derivatives (model.f90:363-401)
//   k_hs_pairs    per atom pair: two-body sum over the translations from the
//                 family's damping kernel (damping.f90:393-539) and the ATM sum
//                 (atm.f90:38-429) over all third atoms: the pair's block of H, of
//                 A = d2E/dR dCN [3N][N] and of D = d2E/dCN2 [N][N], its share of dE/dCN
//   k_hs_diag     dE/dCN and the diagonals of A and D
//   k_hs_cn_hess  the CN second derivative weighted by dE/dCN (ncoord.f90:230-306) and
//                 the diagonal blocks of H
//   k_hs_xyt, k_hs_sym   H += A B^T + B A^T + B D B^T (disp.f90:299-301) as
//                 M B^T + B M^T with M = A + B D / 2
//
// Every off-diagonal block is the sum of one warp, and the diagonals follow from
// translational invariance (H_aa = -sum_b H_ab, A_mm = -sum_a A_am, the same for B),
// so there are no atomics and the result repeats bit for bit.  The work partition
// splits pairs and triples by their owners as the reference does.  O(N^2) memory.
#include <cfloat>
#include <cstdint>

#include "d3_device.cuh"

namespace d3 {

namespace {

constexpr int kHsThreads = 128;
constexpr double kKcnH = 16.0;        // ncoord.f90:31
constexpr double kWfH = 4.0;          // model.f90:80

struct HsSys {
    int n = 0, nid = 0;
    const double* pos = nullptr;      // [n][3] input order
    const int* sp = nullptr;          // [n] species
    const int* zid = nullptr;         // [n] species index inside the structure, from 1
    const uint8_t* ghost = nullptr;   // [n] or null
    const double* img = nullptr;      // lattice translations
    int img_cn0 = 0, img_cn1 = 0, img2_0 = 0, img2_1 = 0, img3_0 = 0, img3_1 = 0;
};

__device__ __forceinline__ bool hs_owns(const Partition& p, int i, int j)
{
    // partition.f90:127-147 on input indices
    if (p.nparts <= 1) return true;
    long long hi = i > j ? i : j, lo = i > j ? j : i;
    return (hi * (hi + 1) / 2 + lo) % p.nparts == p.part;
}

// pair (i, j <= i) of thread t in a lower-triangle sweep of n atoms; false
// beyond the triangle (one thread per matrix element)
__device__ __forceinline__ bool hs_pair(long long t, int n, int& i, int& j)
{
    i = (int)(t / n);
    j = (int)(t % n);
    return i < n && j <= i;
}

__device__ __forceinline__ double hs_wsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per atom m, the lanes over the partners.
__global__ void __launch_bounds__(kHsThreads)
k_hs_cn(HsSys h, Species s, double cutoff, double* B, double* gw, double* dgw, double* d2gw)
{
    const int lane = threadIdx.x & 31;
    const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (m >= h.n) return;
    const int n = h.n;
    const double cut2 = cutoff * cutoff;
    double c = 0.0, gs[3] = {0.0, 0.0, 0.0};
    for (int a = lane; a < n; a += 32) {
        const double rc = s.rcov[h.sp[m]] + s.rcov[h.sp[a]];
        double g[3] = {0.0, 0.0, 0.0};
        for (int t = h.img_cn0; t < h.img_cn1; t++) {
            double v[3];
            for (int k = 0; k < 3; k++) v[k] = h.pos[3 * m + k] - (h.pos[3 * a + k] + h.img[3 * t + k]);
            const double r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            if (r2 > cut2 || r2 < 1.0e-12) continue;
            const double r1 = sqrt(r2);
            const double cf = 1.0 / (1.0 + exp(-kKcnH * (rc / r1 - 1.0)));
            c += cf;
            if (a == m) continue;
            const double dcf = -cf * (1.0 - cf) * kKcnH * rc / r2;
            for (int k = 0; k < 3; k++) g[k] += dcf * v[k] / r1;
        }
        if (a != m)
            for (int k = 0; k < 3; k++) {
                B[(size_t)(3 * a + k) * n + m] = -g[k];
                gs[k] += g[k];
            }
    }
    const double cn = hs_wsum(c);
    for (int k = 0; k < 3; k++) {
        const double g = hs_wsum(gs[k]);
        if (lane == 0) B[(size_t)(3 * m + k) * n + m] = g;
    }
    // reference weights: lane r takes reference r, the sums run in reference order
    const int sp = h.sp[m];
    const int nref = s.nref[sp];
    const double* cnref = s.refcn + sp * kMaxRef;
    const double wf2 = 2.0 * kWfH;
    const double ref = lane < nref ? cnref[lane] : 0.0;
    const double dcn = ref - cn;
    const double expw = lane < nref ? exp(-kWfH * dcn * dcn) : 0.0;
    double norm = 0.0, dnorm = 0.0, d2norm = 0.0, maxcn = cnref[0];
    for (int r = 0; r < nref; r++) {
        const double e = __shfl_sync(0xffffffffu, expw, r), dr = __shfl_sync(0xffffffffu, dcn, r);
        norm += e;
        dnorm += wf2 * dr * e;
        d2norm += (wf2 * wf2 * dr * dr - wf2) * e;
        maxcn = fmax(maxcn, cnref[r]);
    }
    norm = 1.0 / norm;
    if (lane >= kMaxRef) return;
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    if (lane < nref) {
        const double expd = wf2 * dcn * expw, expdd = (wf2 * wf2 * dcn * dcn - wf2) * expw;
        g0 = expw * norm;
        if (isnan(g0) || isinf(g0)) g0 = maxcn == ref ? 1.0 : 0.0;
        g1 = expd * norm - expw * dnorm * norm * norm;
        if (isnan(g1) || isinf(g1)) g1 = 0.0;
        g2 = expdd * norm - 2.0 * expd * dnorm * norm * norm - expw * d2norm * norm * norm
           + 2.0 * expw * dnorm * dnorm * norm * norm * norm;
        if (isnan(g2) || isinf(g2)) g2 = 0.0;
    }
    gw[m * kMaxRef + lane] = g0;
    dgw[m * kMaxRef + lane] = g1;
    d2gw[m * kMaxRef + lane] = g2;
}

__device__ void hs_smooth_r2(double r2, double cutoff, double width, double& sw, double& dsw, double& d2sw)
{
    // cutoff.f90:104-134
    const double r1 = sqrt(r2);
    double dswdr = 0.0, d2swdr2 = 0.0;
    sw = 1.0;
    if (width > 0.0 && width < cutoff) {
        if (r1 >= cutoff) {
            sw = 0.0;
        } else if (r1 > cutoff - width) {
            const double x = (cutoff - r1) / width;
            sw = x * x * x * (10.0 + x * (-15.0 + 6.0 * x));
            dswdr = -30.0 * x * x * (1.0 - x) * (1.0 - x) / width;
            d2swdr2 = 60.0 * x * (1.0 - x) * (1.0 - 2.0 * x) / (width * width);
        }
    }
    dsw = 0.5 * dswdr / r1;
    d2sw = 0.25 * (d2swdr2 - dswdr / r1) / r2;
}

// element (i, j) of each matrix at [i*n + j]: c6, dC6/dCN_i, d2C6/dCN_i^2 and
// the mixed d2C6/dCN_i dCN_j
// and, for one lattice point, the three-body pair factors {m, P}
__global__ void k_hs_c6(HsSys h, Species s, const double* gw, const double* dgw, const double* d2gw, double* c6,
                        double* dc6, double* d2c6, double* d2mix, double2* mp, Config c, double alp3)
{
    int i, j;
    if (!hs_pair(blockIdx.x * (long long)blockDim.x + threadIdx.x, h.n, i, j)) return;
    const int n = h.n;
    double v = 0, di = 0, dj = 0, d2i = 0, d2j = 0, dm = 0;
    if (!(h.ghost && (h.ghost[i] || h.ghost[j]))) {
        const int si = h.sp[i], sj = h.sp[j];
        const double* ref = s.c6ref + (size_t)(si * h.nid + sj) * kMaxRef * kMaxRef;
        for (int ir = 0; ir < s.nref[si]; ir++)
            for (int jr = 0; jr < s.nref[sj]; jr++) {
                const double rc6 = ref[ir * kMaxRef + jr];
                const double gi = gw[i * kMaxRef + ir], gj = gw[j * kMaxRef + jr];
                const double dgi = dgw[i * kMaxRef + ir], dgj = dgw[j * kMaxRef + jr];
                v += gi * gj * rc6;
                di += dgi * gj * rc6;
                dj += gi * dgj * rc6;
                d2i += d2gw[i * kMaxRef + ir] * gj * rc6;
                d2j += gi * d2gw[j * kMaxRef + jr] * rc6;
                dm += dgi * dgj * rc6;
            }
    }
    c6[(size_t)i * n + j] = v; c6[(size_t)j * n + i] = v;
    dc6[(size_t)i * n + j] = di; dc6[(size_t)j * n + i] = dj;
    d2c6[(size_t)i * n + j] = d2i; d2c6[(size_t)j * n + i] = d2j;
    d2mix[(size_t)i * n + j] = dm; d2mix[(size_t)j * n + i] = dm;
    if (!mp || i == j) return;
    double x = 0.0;
    for (int k = 0; k < 3; k++) {
        const double t = h.pos[3 * i + k] - h.pos[3 * j + k];
        x += t * t;
    }
    double2 f = make_double2(0.0, 0.0);
    if (!(x > c.cut3 * c.cut3 || x < DBL_EPSILON)) {
        const double u = 1.0 / x, r0 = s.atm_r0[h.sp[i] * h.nid + h.sp[j]];
        f.x = fabs(v) < DBL_EPSILON ? 0.0 : sqrt(fabs(v)) * u * sqrt(u);
        f.y = fmin(exp(0.5 * alp3 * log(r0 * r0 * u)), 1e100);
        if (c.width3 > 0.0) {
            double sw, d1, d2;
            hs_smooth_r2(x, c.cut3, c.width3, sw, d1, d2);
            f.x *= sw;
        }
    }
    mp[(size_t)i * n + j] = f;
    mp[(size_t)j * n + i] = f;
}

// The family's pair kernel (get_damping_kernel of rational, zero, mzero,
// optimizedpower, cso and z.f90): e = -C6 p(u), u = r^2, and e_u, e_c,
// e_uu, e_uc, e_cc.
__device__ void hs_damping_kernel(const Damp& d, double rrij, double rvdw, int zsum, double u, double c6,
                                  double k[6])
{
    for (int q = 0; q < 6; q++) k[q] = 0.0;
    if (d.kind != kCSO && fabs(d.s6) < DBL_EPSILON && fabs(d.s8) < DBL_EPSILON) return;
    double pv, pd, pdd, pc = 0.0, puc = 0.0, pcc = 0.0;
    if (d.kind == kRational) {
        const double r0 = d.a1 * sqrt(rrij) + d.a2, r02 = r0 * r0, r06 = r02 * r02 * r02, r08 = r06 * r02;
        const double t6 = 1.0 / (u * u * u + r06), t8 = 1.0 / (u * u * u * u + r08);
        const double t6d = -3.0 * u * u * t6 * t6, t8d = -4.0 * u * u * u * t8 * t8;
        const double t6dd = -6.0 * u * t6 * t6 + 18.0 * (u * u * u * u) * (t6 * t6 * t6);
        const double t8dd = -12.0 * u * u * t8 * t8 + 32.0 * (u * u * u * u * u * u) * (t8 * t8 * t8);
        pv = d.s6 * t6 + d.s8 * rrij * t8;
        pd = d.s6 * t6d + d.s8 * rrij * t8d;
        pdd = d.s6 * t6dd + d.s8 * rrij * t8dd;
    } else if (d.kind == kZero || d.kind == kMZero) {
        const double alp6 = d.alp, alp8 = d.alp + 2.0;
        double t6, t8, t6d, t8d, t6dd, t8dd;
        if (d.kind == kZero) {
            const double a6 = 0.5 * alp6, a8 = 0.5 * alp8;
            t6 = pow(d.rs6 * rvdw / sqrt(u), alp6);
            t8 = pow(d.rs8 * rvdw / sqrt(u), alp8);
            t6d = -a6 * t6 / u;
            t8d = -a8 * t8 / u;
            t6dd = a6 * (a6 + 1.0) * t6 / (u * u);
            t8dd = a8 * (a8 + 1.0) * t8 / (u * u);
        } else {
            const double r1 = sqrt(u), betr0 = d.bet * rvdw;
            const double w6 = r1 / (d.rs6 * rvdw) + betr0, w8 = r1 / (d.rs8 * rvdw) + betr0;
            const double w6d = 1.0 / (d.rs6 * rvdw * 2.0 * r1), w8d = 1.0 / (d.rs8 * rvdw * 2.0 * r1);
            const double w6dd = -1.0 / (d.rs6 * rvdw * 4.0 * u * r1), w8dd = -1.0 / (d.rs8 * rvdw * 4.0 * u * r1);
            t6 = pow(w6, -alp6);
            t8 = pow(w8, -alp8);
            t6d = -alp6 * pow(w6, -alp6 - 1.0) * w6d;
            t8d = -alp8 * pow(w8, -alp8 - 1.0) * w8d;
            t6dd = alp6 * (alp6 + 1.0) * pow(w6, -alp6 - 2.0) * w6d * w6d - alp6 * pow(w6, -alp6 - 1.0) * w6dd;
            t8dd = alp8 * (alp8 + 1.0) * pow(w8, -alp8 - 2.0) * w8d * w8d - alp8 * pow(w8, -alp8 - 1.0) * w8dd;
        }
        const double f6 = 1.0 / (1.0 + 6.0 * t6), f8 = 1.0 / (1.0 + 6.0 * t8);
        const double f6d = -6.0 * t6d * f6 * f6, f8d = -6.0 * t8d * f8 * f8;
        const double f6dd = -6.0 * t6dd * f6 * f6 + 72.0 * t6d * t6d * (f6 * f6 * f6);
        const double f8dd = -6.0 * t8dd * f8 * f8 + 72.0 * t8d * t8d * (f8 * f8 * f8);
        const double c6t = f6 / (u * u * u), c6td = f6d / (u * u * u) - 3.0 * f6 / (u * u * u * u);
        const double c6tdd = f6dd / (u * u * u) - 6.0 * f6d / (u * u * u * u) + 12.0 * f6 / (u * u * u * u * u);
        const double c8t = f8 / (u * u * u * u), c8td = f8d / (u * u * u * u) - 4.0 * f8 / (u * u * u * u * u);
        const double c8tdd = f8dd / (u * u * u * u) - 8.0 * f8d / (u * u * u * u * u) + 20.0 * f8 / (u * u * u * u * u * u);
        pv = d.s6 * c6t + d.s8 * rrij * c8t;
        pd = d.s6 * c6td + d.s8 * rrij * c8td;
        pdd = d.s6 * c6tdd + d.s8 * rrij * c8tdd;
    } else if (d.kind == kOptimizedPower) {
        const double r0 = d.a1 * sqrt(rrij) + d.a2, r02 = r0 * r0, r06 = r02 * r02 * r02, r08 = r06 * r02;
        const double ab = pow(r0, d.bet), a6 = ab * r06, a8 = ab * r08, q = 0.5 * d.bet;
        const double d6 = (u * u * u) + a6 * pow(u, -q), d8 = (u * u * u * u) + a8 * pow(u, -q);
        const double d6d = 3.0 * u * u - q * a6 * pow(u, -q - 1.0), d8d = 4.0 * (u * u * u) - q * a8 * pow(u, -q - 1.0);
        const double d6dd = 6.0 * u + q * (q + 1.0) * a6 * pow(u, -q - 2.0);
        const double d8dd = 12.0 * u * u + q * (q + 1.0) * a8 * pow(u, -q - 2.0);
        const double t6 = 1.0 / d6, t8 = 1.0 / d8;
        const double t6d = -d6d * t6 * t6, t8d = -d8d * t8 * t8;
        const double t6dd = -d6dd * t6 * t6 + 2.0 * d6d * d6d * (t6 * t6 * t6);
        const double t8dd = -d8dd * t8 * t8 + 2.0 * d8d * d8d * (t8 * t8 * t8);
        pv = d.s6 * t6 + d.s8 * rrij * t8;
        pd = d.s6 * t6d + d.s8 * rrij * t8d;
        pdd = d.s6 * t6dd + d.s8 * rrij * t8dd;
    } else if (d.kind == kCSO) {
        const double r1 = sqrt(u), r0 = sqrt(rrij);
        const double dd6_6 = pow(d.rs6 * r0 + d.rs8, 6);
        const double sf = 1.0 / (1.0 + exp(r1 - d.a2 * r0));
        const double sfd = -sf * (1.0 - sf), sfdd = sf * (1.0 - sf) * (1.0 - 2.0 * sf);
        const double sig = d.s6 + d.a1 * sf, sigd = d.a1 * sfd, sigdd = d.a1 * sfdd;
        const double sigu = 0.5 * sigd / r1, siguu = 0.25 * sigdd / u - 0.25 * sigd / (u * r1);
        const double t6 = 1.0 / (u * u * u + dd6_6);
        const double t6d = -3.0 * u * u * t6 * t6, t6dd = -6.0 * u * t6 * t6 + 18.0 * (u * u * u * u) * (t6 * t6 * t6);
        pv = sig * t6;
        pd = sigu * t6 + sig * t6d;
        pdd = siguu * t6 + 2.0 * sigu * t6d + sig * t6dd;
    } else {
        const double r0 = d.a1 / double(zsum), b8 = r0 * rrij;
        const double t6 = 1.0 / (u * u * u + r0 * c6), t8 = 1.0 / (u * u * u * u + b8 * c6);
        const double t6u = -3.0 * u * u * t6 * t6, t8u = -4.0 * (u * u * u) * t8 * t8;
        const double t6uu = -6.0 * u * t6 * t6 + 18.0 * (u * u * u * u) * (t6 * t6 * t6);
        const double t8uu = -12.0 * u * u * t8 * t8 + 32.0 * (u * u * u * u * u * u) * (t8 * t8 * t8);
        const double t6c = -r0 * t6 * t6, t8c = -b8 * t8 * t8;
        const double t6uc = 6.0 * u * u * r0 * (t6 * t6 * t6), t8uc = 8.0 * (u * u * u) * b8 * (t8 * t8 * t8);
        const double t6cc = 2.0 * r0 * r0 * (t6 * t6 * t6), t8cc = 2.0 * b8 * b8 * (t8 * t8 * t8);
        pv = d.s6 * t6 + d.s8 * rrij * t8;
        pd = d.s6 * t6u + d.s8 * rrij * t8u;
        pdd = d.s6 * t6uu + d.s8 * rrij * t8uu;
        pc = d.s6 * t6c + d.s8 * rrij * t8c;
        puc = d.s6 * t6uc + d.s8 * rrij * t8uc;
        pcc = d.s6 * t6cc + d.s8 * rrij * t8cc;
    }
    k[0] = -c6 * pv;
    k[1] = -c6 * pd;
    k[2] = -pv - c6 * pc;
    k[3] = -c6 * pdd;
    k[4] = -pd - c6 * puc;
    k[5] = -2.0 * pc - c6 * pcc;
}

struct HsMats {
    const double *c6, *dc6, *d2c6, *d2mix;   // [n][n]
    const double2* mp;                       // [n][n] {m, P} of the pairs (one lattice point), or null
    double *H;                               // [3n][3n]
    double *A;                               // [3n][n]
    double *D;                               // [n][n]
    double *de, *ds;                         // [n][n] dE/dCN_a and d2E/dCN_a2 shares of partner b
    double *dEdcn;                           // [n]
};

// Factors of one pair of a triple as functions of x = r^2 (d3_atm.cu): u = 1/x,
// m = sqrt(C6) x^-3/2 sw, P = (r0/r)^alp3, L = dln(m)/dx and L' = dL/dx.
struct HsFactor { double u, m, P, L, dL; };

__device__ __forceinline__ HsFactor hs_factor(double x, double c6, double r0, double alp3, const Config& c,
                                              const double2* mp)
{
    HsFactor f;
    f.u = 1.0 / x;
    f.L = -1.5 * f.u;
    f.dL = 1.5 * f.u * f.u;
    if (mp) {
        const double2 v = *mp;
        f.m = v.x;
        f.P = v.y;
    } else {
        f.m = fabs(c6) < DBL_EPSILON ? 0.0 : sqrt(fabs(c6)) * f.u * sqrt(f.u);
        f.P = fmin(exp(0.5 * alp3 * log(r0 * r0 * f.u)), 1e100);
    }
    if (c.width3 > 0.0) {
        double sw, d1, d2;
        hs_smooth_r2(x, c.cut3, c.width3, sw, d1, d2);
        if (!mp) f.m *= sw;
        if (sw > 0.0) {
            const double l = d1 / sw;
            f.L += l;
            f.dL += d2 / sw - l * l;
        }
    }
    return f;
}

// One warp per atom pair (a, b <= a): all lattice translations of b, and for each
// the third atoms c and their images over the lanes.  With sites a, b and c, pairs
// 1 = ab, 2 = ac, 3 = bc and the derivatives E_p, E_pq of the triple energy with
// respect to their x, the block is
//   H_ab = sum_c -4 E_11 ab ab^T + 4 E_13 ab bc^T - 4 E_12 ac ab^T + 4 E_23 ac bc^T - 2 E_1,
// and with q_s(p) = dlnC6_p/dCN_s the CN derivatives are E (q_s + q_s') / 2: the sums
// over c below carry every block of the pair (a site pair occurs once among all
// (T_b, c, T_c), so triples with images of one atom need no weights).  For a = b only
// the CN derivatives of the image pairs remain, the rest cancels.
//
// What bounds it: FP64 latency (about 250 instructions per third atom and lane, 35
// sums).  One thread per pair (a, b) with 250 FP64 atomics per triple, as before, took
// the call on 73 atoms 1.52 ms; a triple is now evaluated three times, once per pair,
// without atomics: 0.26 ms, of which this kernel is 0.04 ms.
__global__ void __launch_bounds__(kHsThreads) k_hs_pairs(HsSys h, Species s, Damp d, Config c, Partition part,
                                                         const double* rvdw, HsMats m, int threebody)
{
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int n = h.n;
    if (w >= (long long)n * (n + 1) / 2) return;
    int a = (int)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
    while ((long long)(a + 1) * (a + 2) / 2 <= w) a++;
    while ((long long)a * (a + 1) / 2 > w) a--;
    const int b = (int)(w - (long long)a * (a + 1) / 2);
    const bool self = a == b;
    const int sa = h.sp[a], sb = h.sp[b];
    const double pa[3] = {h.pos[3 * a], h.pos[3 * a + 1], h.pos[3 * a + 2]};
    const double pb[3] = {h.pos[3 * b], h.pos[3 * b + 1], h.pos[3 * b + 2]};
    const double c6ab = m.c6[(size_t)a * n + b];
    const double da = m.dc6[(size_t)a * n + b], db = m.dc6[(size_t)b * n + a];
    const double d2a = m.d2c6[(size_t)a * n + b], d2b = m.d2c6[(size_t)b * n + a], dm = m.d2mix[(size_t)a * n + b];
    // results of the pair
    double Hab[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, Aab[3] = {0, 0, 0}, Aba[3] = {0, 0, 0};
    double Dab = 0, Sa = 0, Sb = 0, ea = 0, eb = 0;

    // ---- two-body: the lanes take the translations
    if (hs_owns(part, a, b)) {
        const double rrij = s.pair[kPairSlots * (sa * h.nid + sb)];
        const double r0 = rvdw[sb * h.nid + sa];
        const int zsum = h.zid[a] + h.zid[b];
        const double cut2 = c.cut2 * c.cut2, fac = self ? 0.5 : 1.0;
        double blk[6] = {0, 0, 0, 0, 0, 0}, fcs = 0.0, fccs = 0.0, av[3] = {0, 0, 0};
        for (int t = h.img2_0 + lane; t < h.img2_1; t += 32) {
            double v[3];
            for (int k = 0; k < 3; k++) v[k] = pa[k] - (pb[k] + h.img[3 * t + k]);
            const double r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            if (r2 > cut2 || r2 < DBL_EPSILON) continue;
            double k6[6], sw, swr, swrr;
            hs_damping_kernel(d, rrij, r0, zsum, r2, c6ab, k6);
            hs_smooth_r2(r2, c.cut2, c.width2, sw, swr, swrr);
            const double fr = fac * (swr * k6[0] + sw * k6[1]);
            const double frr = fac * (swrr * k6[0] + 2.0 * swr * k6[1] + sw * k6[3]);
            const double frc = fac * (swr * k6[2] + sw * k6[4]);
            if (!self) {
                blk[0] += 4.0 * frr * v[0] * v[0] + 2.0 * fr;
                blk[1] += 4.0 * frr * v[1] * v[1] + 2.0 * fr;
                blk[2] += 4.0 * frr * v[2] * v[2] + 2.0 * fr;
                blk[3] += 4.0 * frr * v[0] * v[1];
                blk[4] += 4.0 * frr * v[0] * v[2];
                blk[5] += 4.0 * frr * v[1] * v[2];
                for (int k = 0; k < 3; k++) av[k] += 2.0 * frc * v[k];
            }
            fcs += fac * sw * k6[2];
            fccs += fac * sw * k6[5];
        }
        fcs = hs_wsum(fcs);
        fccs = hs_wsum(fccs);
        if (self) {
            // C6_aa depends on CN_a twice
            ea += 2.0 * fcs * da;
            Sa += 4.0 * fccs * da * da + fcs * (2.0 * d2a + 2.0 * dm);
        } else {
            for (int k = 0; k < 6; k++) blk[k] = hs_wsum(blk[k]);
            for (int k = 0; k < 3; k++) {
                av[k] = hs_wsum(av[k]);
                Aab[k] += av[k] * db;
                Aba[k] -= av[k] * da;
                Hab[k][k] -= blk[k];
            }
            Hab[0][1] -= blk[3]; Hab[1][0] -= blk[3];
            Hab[0][2] -= blk[4]; Hab[2][0] -= blk[4];
            Hab[1][2] -= blk[5]; Hab[2][1] -= blk[5];
            ea += fcs * da;
            eb += fcs * db;
            Sa += fccs * da * da + fcs * d2a;
            Sb += fccs * db * db + fcs * d2b;
            Dab += fccs * da * db + fcs * dm;
        }
    }

    // ---- three-body
    if (threebody && fabs(c6ab) >= DBL_EPSILON) {
        const double cut2 = c.cut3 * c.cut3, alp3 = (d.alp + 2.0) / 3.0, hx = 0.5 * alp3;
        const double ic6 = 1.0 / c6ab, qa1 = da * ic6, qb1 = db * ic6;
        const double r0ab = s.atm_r0[sa * h.nid + sb];
        const int nT = h.img3_1 - h.img3_0;
        for (int tb = 0; tb < nT; tb++) {
            double v1[3];
            for (int k = 0; k < 3; k++) v1[k] = pb[k] + h.img[3 * (h.img3_0 + tb) + k] - pa[k];
            const double x1 = v1[0] * v1[0] + v1[1] * v1[1] + v1[2] * v1[2];
            if (x1 > cut2 || x1 < DBL_EPSILON) continue;
            const HsFactor f1 = hs_factor(x1, c6ab, r0ab, alp3, c, m.mp ? m.mp + (size_t)a * n + b : nullptr);
            // sums over the third atoms
            double W = 0, Xa = 0, Xb = 0, Y = 0;
            double s1 = 0, s11 = 0, s1a = 0, s1b = 0;
            double s12[3] = {0, 0, 0}, s13[3] = {0, 0, 0}, s2[3] = {0, 0, 0}, s3[3] = {0, 0, 0};
            double s2b[3] = {0, 0, 0}, s3a[3] = {0, 0, 0}, s23[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int e = lane; e < n * nT; e += 32) {
                const int cc = nT == 1 ? e : e / nT, tc = e - cc * nT;
                if (part.nparts > 1) {
                    // owner of the triple: the pair of its two largest indices
                    const int lo2 = cc > a ? a : (cc > b ? cc : b);
                    if (!hs_owns(part, cc > a ? cc : a, lo2)) continue;
                }
                double v2[3], v3[3];
                for (int k = 0; k < 3; k++) {
                    v2[k] = h.pos[3 * cc + k] + h.img[3 * (h.img3_0 + tc) + k] - pa[k];
                    v3[k] = v2[k] - v1[k];
                }
                const double x2 = v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2];
                const double x3 = v3[0] * v3[0] + v3[1] * v3[1] + v3[2] * v3[2];
                if (x2 > cut2 || x2 < DBL_EPSILON || x3 > cut2 || x3 < DBL_EPSILON) continue;
                const double c2 = m.c6[(size_t)cc * n + a], c3 = m.c6[(size_t)cc * n + b];
                if (fabs(c2) < DBL_EPSILON || fabs(c3) < DBL_EPSILON) continue;
                const int sc = h.sp[cc];
                const HsFactor f2 = hs_factor(x2, c2, s.atm_r0[sa * h.nid + sc], alp3, c,
                                              m.mp ? m.mp + (size_t)cc * n + a : nullptr);
                const HsFactor f3 = hs_factor(x3, c3, s.atm_r0[sb * h.nid + sc], alp3, c,
                                              m.mp ? m.mp + (size_t)cc * n + b : nullptr);
                const double mm = d.s9 * f1.m * f2.m * f3.m;
                const double cU = 0.375 * f1.u * f2.u * f3.u;
                const double f = 1.0 / (1.0 + 6.0 * f1.P * f2.P * f3.P);
                const double a1 = x1 + x3 - x2, a2 = x1 + x2 - x3, a3 = x2 + x3 - x1;
                const double q1 = a1 * a2, q2 = a2 * a3, q3 = a1 * a3;
                const double A = cU * q1 * a3;
                // A_p = cU S_p - u_p A
                const double S1 = cU * (q3 + q2 - q1), S2 = cU * (q3 - q2 + q1), S3 = cU * (q2 - q3 + q1);
                const double A1 = S1 - f1.u * A, A2 = S2 - f2.u * A, A3 = S3 - f3.u * A;
                const double A11 = cU * (2.0 * a3 - 4.0 * x1) - 2.0 * f1.u * A1;
                const double A12 = cU * 2.0 * a2 - f2.u * S1 - f1.u * A2;
                const double A13 = cU * 2.0 * a1 - f3.u * S1 - f1.u * A3;
                const double A23 = cU * 2.0 * a3 - f3.u * S2 - f2.u * A3;
                // f_p = hx u_p f (1 - f)
                const double ph = hx * f * (1.0 - f), p2 = hx * (1.0 - 2.0 * f) * ph;
                const double F1 = ph * f1.u, F2 = ph * f2.u, F3 = ph * f3.u;
                const double F11 = (p2 - ph) * f1.u * f1.u, F12 = p2 * f1.u * f2.u, F13 = p2 * f1.u * f3.u,
                             F23 = p2 * f2.u * f3.u;
                const double B1 = 1.0 + A, G = B1 * f;
                const double G1 = A1 * f + B1 * F1, G2 = A2 * f + B1 * F2, G3 = A3 * f + B1 * F3;
                const double G11 = A11 * f + 2.0 * A1 * F1 + B1 * F11;
                const double G12 = A12 * f + A1 * F2 + A2 * F1 + B1 * F12;
                const double G13 = A13 * f + A1 * F3 + A3 * F1 + B1 * F13;
                const double G23 = A23 * f + A2 * F3 + A3 * F2 + B1 * F23;
                const double E = mm * G;
                const double qa2 = m.dc6[(size_t)a * n + cc] / c2, qb3 = m.dc6[(size_t)b * n + cc] / c3;
                W += E;
                Xa += E * qa2;
                Xb += E * qb3;
                Y += E * qa2 * qb3;
                if (self) continue;
                const double E1 = mm * (G1 + f1.L * G), E2 = mm * (G2 + f2.L * G), E3 = mm * (G3 + f3.L * G);
                const double E11 = mm * (G11 + 2.0 * f1.L * G1 + (f1.L * f1.L + f1.dL) * G);
                const double E12 = mm * (G12 + f1.L * G2 + f2.L * G1 + f1.L * f2.L * G);
                const double E13 = mm * (G13 + f1.L * G3 + f3.L * G1 + f1.L * f3.L * G);
                const double E23 = mm * (G23 + f2.L * G3 + f3.L * G2 + f2.L * f3.L * G);
                s1 += E1;
                s11 += E11;
                s1a += E1 * qa2;
                s1b += E1 * qb3;
                for (int k = 0; k < 3; k++) {
                    s12[k] += E12 * v2[k];
                    s13[k] += E13 * v3[k];
                    s2[k] += E2 * v2[k];
                    s3[k] += E3 * v3[k];
                    s2b[k] += qb3 * E2 * v2[k];
                    s3a[k] += qa2 * E3 * v3[k];
                    for (int l = 0; l < 3; l++) s23[3 * k + l] += E23 * v2[k] * v3[l];
                }
            }
            W = hs_wsum(W); Xa = hs_wsum(Xa); Xb = hs_wsum(Xb); Y = hs_wsum(Y);
            ea += 0.5 * qa1 * W;
            Sa += 0.25 * qa1 * (Xa - qa1 * W) + 0.5 * d2a * ic6 * W;
            const double dab = 0.25 * (qa1 * Xb + qb1 * Xa + Y - qa1 * qb1 * W) + 0.5 * dm * ic6 * W;
            if (self) {
                Sa += dab;
                continue;
            }
            eb += 0.5 * qb1 * W;
            Sb += 0.25 * qb1 * (Xb - qb1 * W) + 0.5 * d2b * ic6 * W;
            Dab += dab;
            s1 = hs_wsum(s1); s11 = hs_wsum(s11); s1a = hs_wsum(s1a); s1b = hs_wsum(s1b);
            for (int k = 0; k < 3; k++) {
                s12[k] = hs_wsum(s12[k]); s13[k] = hs_wsum(s13[k]);
                s2[k] = hs_wsum(s2[k]); s3[k] = hs_wsum(s3[k]);
                s2b[k] = hs_wsum(s2b[k]); s3a[k] = hs_wsum(s3a[k]);
            }
            for (int k = 0; k < 9; k++) s23[k] = hs_wsum(s23[k]);
            for (int k = 0; k < 3; k++) {
                for (int l = 0; l < 3; l++)
                    Hab[k][l] += 4.0 * (v1[k] * s13[l] - s12[k] * v1[l] + s23[3 * k + l] - s11 * v1[k] * v1[l]);
                Hab[k][k] -= 2.0 * s1;
                Aab[k] -= (qb1 * s1 + s1b) * v1[k] + qb1 * s2[k] + s2b[k];
                Aba[k] += (qa1 * s1 + s1a) * v1[k] - qa1 * s3[k] - s3a[k];
            }
        }
    }
    if (lane != 0) return;
    m.de[(size_t)a * n + b] = ea;
    m.ds[(size_t)a * n + b] = Sa;
    if (self) return;
    m.de[(size_t)b * n + a] = eb;
    m.ds[(size_t)b * n + a] = Sb;
    m.D[(size_t)a * n + b] = Dab;
    m.D[(size_t)b * n + a] = Dab;
    const size_t n3 = 3 * (size_t)n;
    for (int k = 0; k < 3; k++) {
        m.A[(size_t)(3 * a + k) * n + b] = Aab[k];
        m.A[(size_t)(3 * b + k) * n + a] = Aba[k];
        for (int l = 0; l < 3; l++) {
            m.H[(3 * a + k) * n3 + 3 * b + l] = Hab[k][l];
            m.H[(3 * b + l) * n3 + 3 * a + k] = Hab[k][l];
        }
    }
}

// dE/dCN_a, D_aa (sums over the partners) and A_aa = -sum_b A_ba: one warp per atom.
__global__ void k_hs_diag(int n, HsMats m)
{
    const int lane = threadIdx.x & 31;
    const int a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (a >= n) return;
    double e = 0, dd = 0, g[3] = {0, 0, 0};
    for (int b = lane; b < n; b += 32) {
        e += m.de[(size_t)a * n + b];
        dd += m.ds[(size_t)a * n + b];
        if (b != a)
            for (int k = 0; k < 3; k++) g[k] -= m.A[(size_t)(3 * b + k) * n + a];
    }
    e = hs_wsum(e);
    dd = hs_wsum(dd);
    for (int k = 0; k < 3; k++) g[k] = hs_wsum(g[k]);
    if (lane != 0) return;
    m.dEdcn[a] = e;
    m.D[(size_t)a * n + a] = dd;
    for (int k = 0; k < 3; k++) m.A[(size_t)(3 * a + k) * n + a] = g[k];
}

// Adds the CN second derivatives to the blocks of row a and forms the diagonal
// block: one warp per atom, the lanes over the partners.
__global__ void __launch_bounds__(kHsThreads)
k_hs_cn_hess(HsSys h, Species s, double cutoff, const double* dEdcn, double* H)
{
    const int lane = threadIdx.x & 31;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= h.n) return;
    const size_t n3 = 3 * (size_t)h.n;
    const double cut2 = cutoff * cutoff;
    double diag[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = lane; j < h.n; j += 32) {
        if (j == i) continue;
        const double rc = s.rcov[h.sp[i]] + s.rcov[h.sp[j]];
        const double de = dEdcn[i] + dEdcn[j];
        double blk[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int t = h.img_cn0; t < h.img_cn1; t++) {
            double v[3];
            for (int k = 0; k < 3; k++) v[k] = h.pos[3 * i + k] - (h.pos[3 * j + k] + h.img[3 * t + k]);
            const double r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            if (r2 > cut2 || r2 < 1.0e-12) continue;
            const double r1 = sqrt(r2);
            const double cf = 1.0 / (1.0 + exp(-kKcnH * (rc / r1 - 1.0)));
            const double tmp = cf * (1.0 - cf);
            const double dcf = -tmp * kKcnH * rc / r2;
            const double d2cf = tmp * (1.0 - 2.0 * cf) * (kKcnH * rc) * (kKcnH * rc) / (r2 * r2)
                              + 2.0 * tmp * kKcnH * rc / (r2 * r1);
            for (int a = 0; a < 3; a++) {
                for (int b = 0; b < 3; b++) blk[a][b] += de * (d2cf * v[a] * v[b] / r2 - dcf * v[a] * v[b] / (r2 * r1));
                blk[a][a] += de * dcf / r1;
            }
        }
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                double* o = H + (3 * i + a) * n3 + 3 * j + b;
                const double x = *o - blk[a][b];
                *o = x;
                diag[3 * a + b] -= x;
            }
    }
    for (int k = 0; k < 9; k++) {
        const double x = hs_wsum(diag[k]);
        if (lane == 0) H[(3 * i + k / 3) * n3 + 3 * i + k % 3] = x;
    }
}

// C[r][q] = C0[r][q] + f sum_k X[r][k] Y[q][k] for r < M, q < N, k < K (row-major,
// FP64), 16 x 16 tiles staged in shared memory
constexpr int kXyt = 16;
__global__ void k_hs_xyt(const double* X, const double* Y, const double* C0, double f, double* C, int M, int N, int K,
                         int ldc)
{
    __shared__ double xs[kXyt][kXyt + 1], ys[kXyt][kXyt + 1];
    const int r = blockIdx.y * kXyt + threadIdx.y, q = blockIdx.x * kXyt + threadIdx.x;
    double acc = 0.0;
    for (int k0 = 0; k0 < K; k0 += kXyt) {
        const int kx = k0 + threadIdx.x;
        const int ry = blockIdx.y * kXyt + threadIdx.y, qy = blockIdx.x * kXyt + threadIdx.y;
        xs[threadIdx.y][threadIdx.x] = (ry < M && kx < K) ? X[(size_t)ry * K + kx] : 0.0;
        ys[threadIdx.y][threadIdx.x] = (qy < N && kx < K) ? Y[(size_t)qy * K + kx] : 0.0;
        __syncthreads();
        for (int k = 0; k < kXyt; k++) acc += xs[threadIdx.y][k] * ys[threadIdx.x][k];
        __syncthreads();
    }
    if (r < M && q < N) C[(size_t)r * ldc + q] = C0[(size_t)r * ldc + q] + f * acc;
}

// out = H + X Y^T + Y X^T (H [N][N], X and Y [N][K]), the lower triangle of tiles with
// its mirror image, transposed through shared memory for whole rows of 128 bytes: H is
// symmetric.  out may be H or pinned host memory: the result of 73 atoms arrives with the
// kernel, where a copy to pageable memory took a fifth of the call (247 us, 198 now).
__global__ void k_hs_sym(const double* X, const double* Y, const double* H, double* out, int N, int K)
{
    __shared__ double xr[kXyt][kXyt + 1], yr[kXyt][kXyt + 1], xq[kXyt][kXyt + 1], yq[kXyt][kXyt + 1];
    __shared__ double mirror[kXyt][kXyt + 1];
    if (blockIdx.x > blockIdx.y) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int rt = blockIdx.y * kXyt + ty, qt = blockIdx.x * kXyt + ty;
    double acc = 0.0;
    for (int k0 = 0; k0 < K; k0 += kXyt) {
        const int k = k0 + tx;
        const bool rin = rt < N && k < K, qin = qt < N && k < K;
        xr[ty][tx] = rin ? X[(size_t)rt * K + k] : 0.0;
        yr[ty][tx] = rin ? Y[(size_t)rt * K + k] : 0.0;
        xq[ty][tx] = qin ? X[(size_t)qt * K + k] : 0.0;
        yq[ty][tx] = qin ? Y[(size_t)qt * K + k] : 0.0;
        __syncthreads();
#pragma unroll
        for (int l = 0; l < kXyt; l++) acc += xr[ty][l] * yq[tx][l] + yr[ty][l] * xq[tx][l];
        __syncthreads();
    }
    const int q = blockIdx.x * kXyt + tx;
    const bool in = rt < N && q < N;
    const double v = in ? H[(size_t)rt * N + q] + acc : 0.0;
    if (in) out[(size_t)rt * N + q] = v;
    if (blockIdx.x == blockIdx.y) return;
    mirror[tx][ty] = v;
    __syncthreads();
    const int mr = blockIdx.x * kXyt + ty, mq = blockIdx.y * kXyt + tx;
    if (mr < N && mq < N) out[(size_t)mr * N + mq] = mirror[ty][tx];
}

}  // namespace

size_t hessian_scratch_doubles(int n)
{
    // weights (3 x 7 n), four C6 matrices, {m, P}, dE/dCN, its shares, B, A, D, M
    const size_t nn = (size_t)n * n;
    return 3 * (size_t)kMaxRef * n + 4 * nn + 2 * nn + (size_t)n + 2 * nn + 3 * nn + 3 * nn + nn + 3 * nn + 1;
}

void launch_hessian(const Species& s, const Damp& d, const Config& c, const Partition& p, int n, int nid,
                    const double* pos, const int* sp, const int* zid, const uint8_t* ghost, const double* img,
                    const int img_range[6], const double* rvdw, double* scratch, double* H, double* out,
                    cudaStream_t stream)
{
    if (n <= 0) return;
    HsSys h;
    h.n = n; h.nid = nid; h.pos = pos; h.sp = sp; h.zid = zid; h.ghost = ghost; h.img = img;
    h.img_cn0 = img_range[0]; h.img_cn1 = img_range[1];
    h.img2_0 = img_range[2]; h.img2_1 = img_range[3];
    h.img3_0 = img_range[4]; h.img3_1 = img_range[5];
    const size_t nn = (size_t)n * n;
    double* mp = scratch;                     // first: aligned for vector loads
    double* gw = mp + 2 * nn;
    double* dgw = gw + (size_t)kMaxRef * n;
    double* d2gw = dgw + (size_t)kMaxRef * n;
    double* c6 = d2gw + (size_t)kMaxRef * n;
    double* dc6 = c6 + nn;
    double* d2c6 = dc6 + nn;
    double* d2mix = d2c6 + nn;
    double* dEdcn = d2mix + nn;
    double* de = dEdcn + n;
    double* ds = de + nn;
    double* B = ds + nn;
    double* A = B + 3 * nn;
    double* D = A + 3 * nn;
    double* M = D + nn;
    const bool threebody = std::fabs(d.s9) >= DBL_EPSILON;
    // pair factors once for the one lattice point of molecules; per triple otherwise
    const bool factors = threebody && h.img3_1 - h.img3_0 == 1;
    const unsigned pblocks = (unsigned)((nn + kHsThreads - 1) / kHsThreads);
    const unsigned ablocks = (unsigned)((32 * (size_t)n + kHsThreads - 1) / kHsThreads);
    const unsigned wblocks = (unsigned)((32 * ((size_t)n * (n + 1) / 2) + kHsThreads - 1) / kHsThreads);
    k_hs_cn<<<ablocks, kHsThreads, 0, stream>>>(h, s, c.cut_cn, B, gw, dgw, d2gw);
    k_hs_c6<<<pblocks, kHsThreads, 0, stream>>>(h, s, gw, dgw, d2gw, c6, dc6, d2c6, d2mix,
                                                factors ? reinterpret_cast<double2*>(mp) : nullptr, c,
                                                (d.alp + 2.0) / 3.0);
    HsMats m{c6, dc6, d2c6, d2mix, factors ? reinterpret_cast<const double2*>(mp) : nullptr, H, A, D, de, ds, dEdcn};
    k_hs_pairs<<<wblocks, kHsThreads, 0, stream>>>(h, s, d, c, p, rvdw, m, threebody ? 1 : 0);
    k_hs_diag<<<ablocks, kHsThreads, 0, stream>>>(n, m);
    k_hs_cn_hess<<<ablocks, kHsThreads, 0, stream>>>(h, s, c.cut_cn, dEdcn, H);
    // M[b][k] = A[b][k] + sum_l B[b][l] D[k][l] / 2, then H += M B^T + B M^T
    const int n3 = 3 * n;
    const dim3 block(kXyt, kXyt);
    k_hs_xyt<<<dim3((n + kXyt - 1) / kXyt, (n3 + kXyt - 1) / kXyt), block, 0, stream>>>(B, D, A, 0.5, M, n3, n, n, n);
    k_hs_sym<<<dim3((n3 + kXyt - 1) / kXyt, (n3 + kXyt - 1) / kXyt), block, 0, stream>>>(M, B, H, out, n3, n);
}

}  // namespace d3
