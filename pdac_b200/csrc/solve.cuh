// solve.cuh -- the per-face phase-coupled momentum system of the corrector,
// sized at compile time.
//
// NP is the number of phases (gas + solid classes).  With NP > 0 every loop
// over phases has a constant trip count and is unrolled, so the matrix and
// right-hand side of a face live in registers; NP = 0 keeps the run-time
// phase count (any nsolid up to PDAC_MAXS) with the arrays in local memory.
// The arithmetic, and its order, is the same for every NP.
#pragma once
#include "phys2d.cuh"

namespace pdac {

template <int NP>
struct Sys {
    static constexpr int M = (NP > 0 ? NP : PDAC_MAXP) + 1;  // 1-based rows and columns
};

template <int NP>
__device__ __forceinline__ int nphases(const Prm &P) { return NP > 0 ? NP : P.nph; }

// Gauss-Jordan with plim decoupling, matrix.f:351-391; a, b 1-based
template <int NP, int M>
__device__ __forceinline__ void gauss_jordan_t(const Prm &P, double (&a)[M][M], double (&b)[M]) {
    const int nph = nphases<NP>(P);
#pragma unroll
    for (int l = 2; l <= nph; ++l) {
        if (fabs(a[l][l]) < P.plim[l - 1]) {
#pragma unroll
            for (int ll = 1; ll <= nph; ++ll) {
                a[ll][ll] = a[ll][ll] + a[l][ll];
                a[l][ll] = 0.0;
                a[ll][l] = 0.0;
            }
            b[l] = 0.0;
        }
    }
#pragma unroll
    for (int l = 1; l <= nph; ++l) {
        if (a[l][l] != 0.0) {
            double div = 1.0 / a[l][l];
#pragma unroll
            for (int lj = l + 1; lj <= nph; ++lj) a[l][lj] = a[l][lj] * div;
            // the reference's elimination also visits row l itself, with a
            // multiplier of 0: that changes nothing but a -0 into a 0
            b[l] = b[l] * div + 0.0;
            a[l][l] = 0.0;
#pragma unroll
            for (int li = 1; li <= nph; ++li) {
                if (li == l) continue;
                double amul = a[li][l];
#pragma unroll
                for (int lj = l + 1; lj <= nph; ++lj) a[li][lj] = a[li][lj] - amul * a[l][lj];
                b[li] = b[li] - amul * b[l];
            }
        }
    }
}

// Doubles of one face record (F.fk): the face's interphase terms
// alpha (d0 app(nb) + d1 app(c)) / (d0 + d1) by interphase index, then the
// tilde momenta of its row (gas first), padded to whole 16-byte pairs.
__host__ __device__ constexpr int face_rec(int nph) { return (nph * (nph + 1) / 2 + nph + 1) / 2 * 2; }
// the record of the E/N/T face of cell c along axis q (0 = x, last = z)
template <int NP>
__device__ __forceinline__ double *face_rec_ptr(const Prm &P, const Fld &F, int q, int c) {
    return F.fk + ((size_t)q * P.ncell + c) * face_rec(NP);
}

// The predictor's face solution (iter.f:135-145): the phase matrix of the
// E/N/T face of cell c along dir (matrix.f:38-328), solved
// (matrix.f:351-630), its velocities stored, when the raw face neighbour is
// fluid.  nb = remapped face neighbour, ii = the cell's index along dir.
// Writes the face's record, which the inner loop of either of its cells
// reads for the rest of iter: neither the interphase terms nor the tilde
// momenta change there, and a face between two fluid cells has the same
// terms seen from both.
template <int NP>
__device__ __forceinline__ void face_solve(const Prm &P, const Fld &F, int c, int nb, int raw, int ii, int dir,
                                           double dt) {
    if (!(P.flag[raw] & 1)) return;
    constexpr int M = Sys<NP>::M;
    const int nph = nphases<NP>(P);
    const size_t n = P.ncell;
    const double *dd = dir == 0 ? P.dx : (dir == 1 ? P.dy : P.dz);
    double grav = dir == 0 ? P.gravx : (dir == 1 ? P.gravy : P.gravz);
    const double *app = dir == 0 ? F.appu : (dir == 1 ? F.appv : F.appw);
    const double *rg = dir == 0 ? F.rug : (dir == 1 ? F.rvg : F.rwg);
    const double *rs = dir == 0 ? F.rus : (dir == 1 ? F.rvs : F.rws);
    double alpha = P.alpha, ag = P.alphagrav;
    double a[M][M], b[M];
    double d0 = dd[ii], d1 = dd[ii + 1];
    double inv = dir == 0 ? P.hx[ii] : (dir == 1 ? P.hy[ii] : P.hz[ii]);
    constexpr int RS = NP > 0 ? face_rec(NP) : 2, NA = NP * (NP + 1) / 2;
    double rec[RS];
    if (NP > 0) rec[RS - 1] = 0.0;  // the padding, where there is one
    double pnb = __ldg(F.p + nb), rgpnb = __ldg(F.rgp + nb), rgpc = F.rgp[c];
    double dp = F.p[c] - pnb;
    double ep_f = 1.0;
    if (P.pmodel == 1) ep_f = (d0 * __ldg(F.ep + nb) + d1 * F.ep[c]) * inv;
    const double r1 = __ldg(rg + c);
    if (NP > 0) rec[NA] = r1;
    b[1] = r1 + alpha * dt * inv * 2.0 * ep_f * dp;
    b[1] = b[1] + dt * ag * inv * grav * (d0 * rgpnb + d1 * rgpc);
    a[1][1] = alpha * (d0 * __ldg(app + nb) + d1 * __ldg(app + c)) * inv;
    if (NP > 0) rec[0] = a[1][1];
    a[1][1] = a[1][1] + (d0 * rgpnb + d1 * rgpc) * inv;
#pragma unroll
    for (int l = 2; l <= nph; ++l) {
        double rn = __ldg(F.rlk + (l - 2) * n + nb), rc = F.rlk[(l - 2) * n + c];
        double eps_f = 0.0;
        if (P.pmodel == 1) eps_f = (d0 * rn + d1 * rc) * inv * P.inrl[l - 1];
        const double rl = __ldg(rs + (l - 2) * n + c);
        if (NP > 0) rec[NA + l - 1] = rl;
        b[l] = rl + alpha * dt * inv * 2.0 * eps_f * dp;
        b[l] = b[l] + dt * ag * inv * grav * (d0 * rn + d1 * rc);
        int ls1 = l * (l - 1) / 2;
#pragma unroll
        for (int ll = 1; ll <= l; ++ll) {
            int ls = ls1 + ll;
            double val = alpha * (d0 * __ldg(app + (ls - 1) * n + nb) + d1 * __ldg(app + (ls - 1) * n + c)) * inv;
            if (NP > 0) rec[ls - 1] = val;
            a[l][ll] = val;
            a[ll][l] = val;
        }
        a[l][l] = a[l][l] + (d0 * rn + d1 * rc) * inv;
    }
    if (NP > 0 && F.fk) {
        double2 *w = reinterpret_cast<double2 *>(face_rec_ptr<NP>(P, F, P.d3 ? dir : dir / 2, c));
#pragma unroll
        for (int q = 0; q < RS / 2; ++q) w[q] = make_double2(rec[2 * q], rec[2 * q + 1]);
    }
    gauss_jordan_t<NP>(P, a, b);
    double *g = dir == 0 ? F.ug : (dir == 1 ? F.vg : F.wg);
    double *s = dir == 0 ? F.us : (dir == 1 ? F.vs : F.ws);
    g[c] = b[1];
#pragma unroll
    for (int l = 2; l <= nph; ++l) s[(l - 2) * n + c] = b[l];
}

// value of a stencil slot: the cell's own current value where the (remapped)
// slot index is the cell itself, else the read-only neighbour value
__device__ __forceinline__ double slot(const double *a, int idx, int c, double own) {
    return idx == c ? own : __ldg(a + idx);
}

// set the active-set bit of cell x (one bit per cell, 32 per word)
__device__ __forceinline__ void mark_dirty(unsigned *dirty, int x) { atomicOr(dirty + (x >> 5), 1u << (x & 31)); }

}  // namespace pdac
