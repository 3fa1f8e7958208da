// inner.cuh -- inner_loop of the corrector (iter.f:480-580) on a team of
// lanes per cell.
//
// A team of T lanes (6 in 3D, 4 in 2D) owns one unconverged cell of the
// worklist.  Lane q < NF owns face q of the cell (3D: W, S, B, E, N, T; 2D:
// W, B, E, T): it assembles and solves that face's phase system and computes
// that face's mass fluxes.  The per-cell quantities (pressure adjustment,
// equation of state, volume fractions, continuity residual) are evaluated by
// every lane of the team from the same inputs, so all lanes hold identical
// values and take the same branches; face values reach the other lanes by
// warp shuffles.  Each value is computed with the same operations in the same
// order as the one-thread form, and the cell's state, face velocities and
// fluxes stay in registers until the final store (nothing else touches the
// cell's neighbourhood within a colour phase).
#pragma once
#include <cooperative_groups.h>
#include "kernels3d.cuh"

namespace pdac {

// a load of a value that no thread of the current launch writes: through
// the read-only cache in the one-launch-per-colour-phase form (RO); a plain
// load in the persistent form, where other blocks write it between the
// phases (separated by grid-wide barriers)
template <bool RO>
__device__ __forceinline__ double ldro(const double *p) {
    if (RO) return __ldg(p);
    return *p;
}
// the same for a stencil slot that may be the cell c itself, which this
// launch does write (later, by the lanes of its own team)
template <bool RO>
__device__ __forceinline__ double ldro_self(const double *a, int idx, int c) {
    return idx == c ? a[c] : ldro<RO>(a + idx);
}

// The mass flux through one face (masf + fmas, flux_m.f:47-324) in
// coordinates mirrored about the cell: n is the cell across the face, f the
// one beyond it, o the one on the other side of the cell c.  The reference's
// gradients are differences along the axis; mirroring a W/S/B face flips the
// sign of all three, which an IEEE difference, product and quotient carry
// exactly, so both kinds of face run the same instructions (one division
// instead of one per branch of face side and velocity sign) and give the
// bits of the reference's expressions (a zero may change its sign).
struct FaceGeo {
    double cn, cf, co;  // 2 x reciprocal spacing of (n, c), (f, n), (c, o)
    double iu, id;      // the MUSCL increment for flow out of the cell / into it, signed like the axis
    double r;           // radial factor of x faces in cylindrical 2D, else 1
    bool lim_on;
};

// cs: face velocity; out: it leaves the cell (upwind side c); d*: densities
template <int D>
__device__ __forceinline__ double face_mflux(const Prm &P, const FaceGeo &g, double cs, bool out, double dc,
                                             double dn, double df, double dopp, bool mus) {
    // the donor-cell flux: of 0.5 (cs -+ |cs|) one is cs, the other 0
    double f = cs * (out ? dc : dn);
    if (D == 2) f = f * g.r;
    if (!mus) return f;
    const double gc = g.cn * (dn - dc);
    const double gf = g.cf * (df - dn), go = g.co * (dc - dopp);
    const double num = out ? go : gf;
    const bool nz = gc != 0;
    const double erre = (nz ? num : 0.0) / (nz ? gc : 1.0);
    const double lim = g.lim_on ? limiter(P.lm, erre, P.beta) : 0.0;
    const double upwnd = lim * gc * (out ? g.iu : g.id);
    double t = upwnd * cs;
    if (D == 2) t = t * g.r;
    return f + t;
}

// Loop-invariant part of one face's phase system (matrix.f:38-328) for the
// cell's inner loop: everything that does not depend on the cell's own p,
// ep, rgp and rlk, evaluated once so that the in-loop assembly
// (face_assemble) gives the bits of the predictor's (face_solve): the face's
// record (rec: interphase terms by interphase index, then the tilde momenta
// of its row, gas first) and seven scalars.  Two storage forms: SH = true
// keeps them as 16-byte pairs in this lane's column of a shared [N][KS]
// array (blocks of KS threads), which frees ~50 registers of the inner loop
// for a third resident block per SM and lets the record arrive by
// asynchronous copies; SH = false (the generic phase count, whose array
// would not fit) keeps them in registers.
constexpr int KS = 128;  // threads per block of every kernel running the inner loop

// the seven scalars of FaceK (and one of padding)
enum { FK_PNB = 0, FK_D0EPNB, FK_K1, FK_K2, FK_D1, FK_INV, FK_D0, FK_N };

template <int NP, bool SH>
struct FaceK;

template <int NP>
struct FaceK<NP, false> {
    static constexpr int M = Sys<NP>::M, R = (M * (M - 1) / 2 + M) / 2 * 2;
    double rec_[R], sc_[FK_N + 1];
    __device__ __forceinline__ explicit FaceK(double *) {}
    __device__ __forceinline__ void set(int i, double v) { rec_[i] = v; }
    __device__ __forceinline__ void get(double (&v)[R]) const {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = rec_[i];
    }
    __device__ __forceinline__ double &sc(int q) { return sc_[q]; }
};

template <int NP>
struct FaceK<NP, true> {
    static constexpr int R = face_rec(NP), N = R + FK_N + 1;
    double *s;  // this lane's column: element q at s[q / 2 * 2 * KS + q % 2]
    __device__ __forceinline__ explicit FaceK(double *cols) : s(cols + 2 * (threadIdx.x % KS)) {}
    __device__ __forceinline__ void set(int i, double v) { s[i / 2 * 2 * KS + i % 2] = v; }
    __device__ __forceinline__ void get(double (&v)[R]) const {
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
            const double2 w = *reinterpret_cast<const double2 *>(s + i * 2 * KS);
            v[2 * i] = w.x;
            v[2 * i + 1] = w.y;
        }
    }
    // the record from global memory, 16 bytes at a time past the L1 (no cell
    // of the colour shares a face with another); fetched() ends the wait
    __device__ __forceinline__ void fetch(const double *rec) const {
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(s + i * 2 * KS);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rec + 2 * i) : "memory");
        }
    }
    __device__ __forceinline__ void fetched() const { asm volatile("cp.async.wait_all;" ::: "memory"); }
    __device__ __forceinline__ double &sc(int q) { return s[(R + q) / 2 * 2 * KS + (R + q) % 2]; }
};

// The loop-invariant density stencil of one face's mass fluxes by phase: the
// values of the cells n, f and o of face_mflux.  SH = true keeps them in this
// lane's column of a shared [3 NC][KS] array, as FaceK does.
template <int NC, bool SH>
struct DensK;

template <int NC>
struct DensK<NC, false> {
    double n_[NC], f_[NC], o_[NC];
    __device__ __forceinline__ explicit DensK(double *) {}
    __device__ __forceinline__ double &n(int l) { return n_[l]; }
    __device__ __forceinline__ double &f(int l) { return f_[l]; }
    __device__ __forceinline__ double &o(int l) { return o_[l]; }
};

template <int NC>
struct DensK<NC, true> {
    double *s;  // this lane's column: element q at s[q * KS]
    __device__ __forceinline__ explicit DensK(double *col) : s(col) {}
    __device__ __forceinline__ double &n(int l) { return s[l * KS]; }
    __device__ __forceinline__ double &f(int l) { return s[(NC + l) * KS]; }
    __device__ __forceinline__ double &o(int l) { return s[(2 * NC + l) * KS]; }
};

// Fills K for the face of cell c whose row is held by cell rowc (c itself on
// the plus side, the neighbour on the minus side), by axis q = dir (3D) or
// 0 / 1 (2D): the record through an asynchronous copy, or, where iter keeps
// none (F.fk null or a generic phase count), from the interphase terms and
// tilde momenta.
template <int NP, bool RO, bool SH, class KT>
__device__ __forceinline__ void face_prepare(const Prm &P, const Fld &F, int c, int nb, int rowc, int ii, int dir,
                                             int side, double dt, KT &K) {
    const int nph = nphases<NP>(P);
    const size_t n = P.ncell;
    const double *dd = dir == 0 ? P.dx : (dir == 1 ? P.dy : P.dz);
    const double *hh = dir == 0 ? P.hx : (dir == 1 ? P.hy : P.hz);
    const double d0 = dd[ii], d1 = side > 0 ? dd[ii + 1] : dd[ii - 1];
    const double inv = side > 0 ? hh[ii] : hh[ii - 1];
    bool rec = false;
    if constexpr (SH) {
        if (F.fk) {
            K.fetch(face_rec_ptr<NP>(P, F, P.d3 ? dir : dir / 2, rowc));
            rec = true;
        }
    }
    if (!rec) {
        const double *app = dir == 0 ? F.appu : (dir == 1 ? F.appv : F.appw);
        const double *rg = dir == 0 ? F.rug : (dir == 1 ? F.rvg : F.rwg);
        const double *rs = dir == 0 ? F.rus : (dir == 1 ? F.rvs : F.rws);
        const int nap = nph * (nph + 1) / 2;
#pragma unroll
        for (int ls = 1; ls <= nap; ++ls)
            K.set(ls - 1, P.alpha * (d0 * __ldg(app + (ls - 1) * n + nb) + d1 * __ldg(app + (ls - 1) * n + c)) * inv);
        K.set(nap, __ldg(rg + rowc));
#pragma unroll
        for (int l = 2; l <= nph; ++l) K.set(nap + l - 1, __ldg(rs + (l - 2) * n + rowc));
    }
    K.sc(FK_D0) = d0;
    K.sc(FK_D1) = d1;
    K.sc(FK_INV) = inv;
    K.sc(FK_PNB) = ldro<RO>(F.p + nb);
    K.sc(FK_D0EPNB) = P.pmodel == 1 ? d0 * ldro<RO>(F.ep + nb) : 0.0;
    K.sc(FK_K1) = P.alpha * dt * inv * 2.0;
    K.sc(FK_K2) = dt * P.alphagrav * inv * (dir == 0 ? P.gravx : (dir == 1 ? P.gravy : P.gravz));
}

// the in-loop assembly and solution: K and Dk of the face, the cell's
// current p, ep, rgp and rlk; side +1 for E/N/T, -1 for W/S/B faces
template <int NP, class KT, class DT>
__device__ __forceinline__ void face_assemble(const Prm &P, KT &K, DT &Dk, int side, double pc, double epc,
                                              double rgpc, const double *rlkc, double *v) {
    constexpr int M = Sys<NP>::M;
    const int nph = nphases<NP>(P), nap = nph * (nph + 1) / 2;
    double a[M][M], b[M], rec[KT::R];
    K.get(rec);
    const double d0 = K.sc(FK_D0), d1 = K.sc(FK_D1), inv = K.sc(FK_INV), pnb = K.sc(FK_PNB);
    const double K1 = K.sc(FK_K1), K2 = K.sc(FK_K2);
    double dp = side > 0 ? pc - pnb : pnb - pc;
    double ep_f = 1.0;
    if (P.pmodel == 1) ep_f = (K.sc(FK_D0EPNB) + d1 * epc) * inv;
    b[1] = rec[nap] + K1 * ep_f * dp;
    const double rgf = d0 * Dk.n(0) + d1 * rgpc;
    b[1] = b[1] + K2 * rgf;
    a[1][1] = rec[0] + rgf * inv;
#pragma unroll
    for (int l = 2; l <= nph; ++l) {
        const double rf = d0 * Dk.n(l - 1) + d1 * rlkc[l - 2];
        double eps_f = 0.0;
        if (P.pmodel == 1) eps_f = rf * inv * P.inrl[l - 1];
        b[l] = rec[nap + l - 1] + K1 * eps_f * dp;
        b[l] = b[l] + K2 * rf;
        int ls1 = l * (l - 1) / 2;
#pragma unroll
        for (int ll = 1; ll <= l; ++ll) {
            double val = rec[ls1 + ll - 1];
            a[l][ll] = val;
            a[ll][l] = val;
        }
        a[l][l] = a[l][l] + rf * inv;
    }
    gauss_jordan_t<NP>(P, a, b);
#pragma unroll
    for (int l = 1; l <= nph; ++l) v[l - 1] = b[l];
}

// minimum resident blocks per SM the register allocation must allow: with
// the face terms in shared memory, up to four phases fit 168 registers and
// three blocks per SM without spilling; more phases take two blocks
#ifndef PDAC_INNER_MINB_SMALL
#define PDAC_INNER_MINB_SMALL 3
#endif
#ifndef PDAC_INNER_MINB_LARGE
#define PDAC_INNER_MINB_LARGE 2
#endif
#define PDAC_INNER_MINB(NP) ((NP) > 0 && (NP) <= 4 ? PDAC_INNER_MINB_SMALL : PDAC_INNER_MINB_LARGE)
#ifndef PDAC_INNER_SHD_MAXP
#define PDAC_INNER_SHD_MAXP 6
#endif

// the inner loop's shared memory, allocated at launch (dynamic): FaceK
// columns for up to six phases, then DensK columns up to
// PDAC_INNER_SHD_MAXP phases (34 KB per block at four phases, 54 at six)
template <int NP>
__host__ __device__ constexpr int inner_face_rows() { return (NP > 0 && NP <= 6) ? FaceK<NP, true>::N : 0; }
template <int NP>
__host__ __device__ constexpr int inner_dens_rows() {
    return (NP > 0 && NP <= PDAC_INNER_SHD_MAXP) ? 3 * (Sys<NP>::M - 1) : 0;
}
template <int NP>
__host__ __device__ constexpr size_t inner_smem_bytes() {
    return (size_t)(inner_face_rows<NP>() + inner_dens_rows<NP>()) * KS * sizeof(double);
}
// The most cells of one colour in 32 consecutive ones, whatever their flags: a
// row of nx cells has one on every third i, so 32 cells over rows of at least 5
// have 14 at most (11 where the rows' first and last cells are not fluid, as on
// the meshes of the reference, whose frame is a boundary).
constexpr int WORD_CELLS = 14;
constexpr int SCAN_LIST = 32 * WORD_CELLS;  // a warp's list of the candidates of 32 words
// the sweep loops', which hold the warps' scan lists in the same place
template <int NP>
__host__ __device__ constexpr size_t sweep_smem_bytes(int threads = KS) {
    constexpr size_t lists = KS / 32 * SCAN_LIST * sizeof(int);
    return (size_t)threads / KS * (inner_smem_bytes<NP>() > lists ? inner_smem_bytes<NP>() : lists);
}

// A worklist entry is a cell, with the top bit set for a plain one: a cell
// whose face stencils meet no wall and stay two cells from the mesh's ends
// (k_colour_masks), so that no flag need be read to know its neighbours --
// one dependent trip to L2 less before the values themselves are asked for.
// The next bit is set for a cell that is expected to take several iterations:
// about half the cells take one and half take three, and a cell that took one
// the last time takes three the next, and the other way round (95 of 100 on
// the plumes).  The bits of the expectation follow the active set's words; it
// decides only which cells share a warp.
constexpr int ENTRY_LONG = 1 << 30;
__device__ __forceinline__ int entry_cell(int e) { return e & (ENTRY_LONG - 1); }
__device__ __forceinline__ unsigned *expect_long(const Prm &P, unsigned *dirty) { return dirty + ((unsigned)P.ncell + 31u) / 32u; }

// The inner loop of worklist entry e (outer sweep nit, 1-based) by the team of
// lanes tb .. tb + T - 1 of this warp (lane q of the team owns face q); kcols
// and dcols are the shared FaceK and DensK arrays.  RO as in ldro.
//
// Every lane of the warp makes this call and runs the same instructions to
// the end: a team whose cell has converged stores it and goes on computing
// values that nothing reads (live = false, also for the lanes that own no
// face and for teams without a cell, which take any valid c), so that the
// shuffles take the whole warp and teams never run apart.  What bounds the
// loop is the dependent FP64 chain of an iteration (~1500 cycles of 8.8-cycle
// operations, 76-cycle reciprocals and 127-cycle quotients, measured) and the
// instructions of a warp's teams when they diverge; hence one code path for
// all faces, velocity signs and bracketing states.
template <int NP, int D, bool RO, bool SPLIT>
__device__ __forceinline__ void inner_team_cell(const Prm &P, const Fld &F, double dt, int nit, int e, bool live,
                                                unsigned *dirty, int q, int tb, double *kcols, double *dcols) {
    constexpr unsigned full = 0xffffffffu;
    constexpr int NC = Sys<NP>::M - 1;   // phase capacity
    constexpr bool SH = inner_face_rows<NP>() > 0;   // FaceK in shared memory (22 KB per block at NP = 4, 36 KB at 6)
    constexpr bool SHD = inner_dens_rows<NP>() > 0;  // DensK too (12 KB at NP = 4, 18 KB at NP = 6)
    constexpr int NAX = D == 3 ? 3 : 2;  // axes; lanes q < NAX own the minus faces
    const int nph = nphases<NP>(P), ns = nph - 1;
    const size_t n = P.ncell;
    const int c = entry_cell(e);
    const bool plain = e < 0;
    int i, j, k;
    if (D == 3) ijk_of(P, c, i, j, k);
    else { i = c % P.nx + 1; j = 1; k = c / P.nx + 1; }
    const int *fl = P.flag;
    // ---- this lane's face: axis, side, raw and remapped neighbours -------
    const bool minus = q < NAX;
    const int a = minus ? q : q - NAX;
    const int dir = D == 3 ? a : (a == 0 ? 0 : 2);
    const int ii = dir == 0 ? i : (dir == 1 ? j : k);
    const int nax = dir == 0 ? P.nx : (dir == 1 ? P.ny : P.nz);
    const int stride = dir == 0 ? 1 : (D == 2 ? P.nx : (dir == 1 ? P.nx : P.nx * P.ny));
    // steps to the clamped neighbours along the axis (raw2 / raw3), in face
    // coordinates: n across the face, f beyond it, o on the other side
    const int toward = minus ? ii - 1 : nax - ii;  // cells to the mesh's end across the face
    const int rawnb = minus ? c - stride * min(1, ii - 1) : c + stride * min(1, nax - ii);
    const int rawop = minus ? c + stride * min(1, nax - ii) : c - stride * min(1, ii - 1);
    const int rawfar = minus ? c - stride * min(2, ii - 1) : c + stride * min(2, nax - ii);
    // the remapped neighbours (rem2 / rem3): a wall reads as the cell itself,
    // a wall beyond the neighbour as the neighbour (y: the remapped one), the
    // last cell before the frame repeats the remapped neighbour
    int fnb = FLUID, rn = rawnb, ro = rawop, rf = rawfar;
    bool mus = P.muscl > 0;
    if (!plain) {
        fnb = fl[rawnb];
        rn = is_wallf(fnb) ? c : rawnb;
        ro = is_wallf(fl[rawop]) ? c : rawop;
        rf = toward == 1 ? rn : (is_wallf(fl[rawfar]) ? (dir == 1 ? rn : rawnb) : rawfar);
        mus = mus && fl[c] == FLUID;
    }
    const bool solved = (fnb & 1) != 0;
    const int fcell = minus ? rawnb : c;  // where this face's velocity and fluxes live
    FaceGeo g;
    {
        const double *dd = dir == 0 ? P.dx : (dir == 1 ? P.dy : P.dz);
        const double *hh = dir == 0 ? P.hx : (dir == 1 ? P.hy : P.hz);
        const double hm = 2.0 * hh[ii - 1], hp = 2.0 * hh[ii];
        g.cn = minus ? hm : hp;
        g.co = minus ? hp : hm;
        g.cf = 2.0 * hh[minus ? max(ii - 2, 0) : ii + 1];
        g.iu = 0.5 * dd[ii];
        g.id = minus ? -0.5 * dd[ii - 1] : -0.5 * dd[ii + 1];
        g.r = (D == 2 && dir == 0) ? (minus ? P.rb[i - 1] : P.rb[i]) : 1.0;
        g.lim_on = toward != 1 && fnb == FLUID;
    }
    double *const gvel = dir == 0 ? F.ug : (dir == 1 ? F.vg : F.wg);
    double *const svel = dir == 0 ? F.us : (dir == 1 ? F.vs : F.ws);
    double *const gfa = dir == 0 ? F.rgfe : (dir == 1 ? F.rgfn : F.rgft);
    double vel[NC];
    vel[0] = gvel[fcell];
#pragma unroll
    for (int l = 2; l <= nph; ++l) vel[l - 1] = svel[(l - 2) * n + fcell];
    FaceK<NP, SH> K(kcols);
    if (solved) face_prepare<NP, RO, SH>(P, F, c, rn, fcell, ii, dir, minus ? -1 : +1, dt, K);
    // density stencil of this face's mass fluxes by phase (gas first).  A
    // slot remapped to the cell reads the cell's own current value, except in
    // opt_inner_loop (iter.f:1255-1547), which builds the stencils once and
    // updates only their centre: there it keeps the loop-entry value, which
    // is what this load reads
    const bool stale = P.opt == 2;
    const bool sn = !stale && rn == c, so = !stale && ro == c, sf = !stale && rf == c, self = sn || so || sf;
    DensK<NC, SHD> Dk(dcols + threadIdx.x % KS);
#pragma unroll
    for (int l = 1; l <= nph; ++l) {
        const double *D_ = l == 1 ? F.rgp : F.rlk + (size_t)(l - 2) * n;
        Dk.n(l - 1) = ldro_self<RO>(D_, rn, c);
        Dk.o(l - 1) = ldro_self<RO>(D_, ro, c);
        Dk.f(l - 1) = mus ? ldro_self<RO>(D_, rf, c) : 0.0;
    }
    auto mflux = [&](int ph, double own) {
        double dn = Dk.n(ph), df = Dk.f(ph), dopp = Dk.o(ph);
        if (self) {
            if (sn) dn = own;
            if (so) dopp = own;
            if (sf) df = own;
        }
        const double cs = vel[ph];
        return face_mflux<D>(P, g, cs, (cs >= 0) != minus, own, dn, df, dopp, mus);
    };
    // ---- cell state (identical in every lane) ------------------------------
    const double rx = D == 2 ? P.inr[i] : 1.0;
    const double idx_i = P.indx[i], idz_k = P.indz[k], idy_j = D == 3 ? P.indy[j] : 0.0;
    const double rgpn_c = F.rgpn[c];
    double bq = 1.0, ivf = 1.0;  // this face's open factor and 1 / fluid fraction (faces, iter.f:259)
    if (P.immb) {
        const int bit = dir == 0 ? (minus ? 2 : 1) : (dir == 1 ? (minus ? 32 : 16) : (minus ? 8 : 4));
        bq = (__ldg(P.ib_faces + c) & bit) ? 1.0 : 0.0;
        ivf = __ldg(P.ib_ivf + c);
    }
    const double dti = dt * ivf;
    // the flux divergence of one phase: every lane gets the axis differences
    // (plus face minus minus face, each times its open factor) over the cell
    // sizes and sums them in the reference's order (x, y, z)
    const double ida = dir == 0 ? idx_i : (dir == 1 ? idy_j : idz_k);
    const int lmin = minus ? q + tb : q - NAX + tb;  // the minus face's lane of this lane's axis
    auto diverg = [&](double fl_) {
        const double w = bq * fl_;
        double d = (w - __shfl_sync(full, w, lmin)) * ida;
        if (D == 2 && dir == 0) d = d * rx;
        const double dx_ = __shfl_sync(full, d, tb + NAX);
        const double dz_ = __shfl_sync(full, d, tb + 2 * NAX - 1);
        const double dy_ = D == 3 ? __shfl_sync(full, d, tb + NAX + 1) : 0.0;
        return D == 3 ? dx_ + dy_ + dz_ : dx_ + dz_;
    };
    // calc_res of the stored state (iter.f:743-771, which sums x + y + z)
    double dg = F.rgp[c] - rgpn_c + dti * diverg(gfa[fcell]);
    double dgorig = dg;
    const double conv = F.conv[c];
    double d3 = dg, p3 = F.p[c], abeta = F.abeta[c];
    // the mixture molecular weight of thermal_eosg (eosg.f:114-137), which
    // does not change within the loop: summed once, in thermal_eosg's order
    double mg = 0;
    for (int ig = 0; ig < P.ng; ++ig) mg = mg + GAS(F.xgc, c, ig) * P.gmw[P.gas_type[ig]];
    const pdac_fp::Recip rgas_tg = pdac_fp::recip(P.rgas * F.tg[c]);
    int kros = -1;
    PAdj s = {0, 0, 0, 0, 0, 0};
    double p = p3, ep = F.ep[c], rog, rgp;
    double rlk[NC], rlkn[NC], snk[NC];
#pragma unroll
    for (int is = 1; is <= ns; ++is) {
        rlk[is - 1] = F.rlk[(is - 1) * n + c];
        rlkn[is - 1] = F.rlkn[(is - 1) * n + c];
        snk[is - 1] = dti * F.sink[(is - 1) * n + c];
    }
    double flux[NC];  // this lane's face mass flux by phase (gas first)
#pragma unroll
    for (int l = 0; l < NC; ++l) flux[l] = 0.0;
    if constexpr (SH) K.fetched();
    for (int loop = 1; loop <= P.inmax; ++loop) {
        if (loop > 1 || nit > 1) padjust(s, p, kros, d3, p3, P.omega, abeta);
        rog = pdac_fp::div_by(p, rgas_tg) * mg;  // thermal_eosg
        rgp = ep * rog;
        // this lane's face system (matrix.f:351-630)
        if (solved) face_assemble<NP>(P, K, Dk, minus ? -1 : +1, p, ep, rgp, rlk, vel);
        // particle mass fluxes and volume fractions (iter.f:778-994)
#pragma unroll
        for (int is = 1; is <= ns; ++is) flux[is] = mflux(is, rlk[is - 1]);
        double rls = 0;
#pragma unroll
        for (int is = 1; is <= ns; ++is) {
            double t = rlkn[is - 1] - dti * diverg(flux[is]);
            t = t + snk[is - 1];
            double v = fmax(0.0, t);
            rlk[is - 1] = v;
            rls = rls + v * P.inrl[is];
        }
        ep = 1.0 - rls;
        if (rls > 1.0 && q == 0 && live) atomicAdd(&F.counters[2], 1);
        rgp = ep * rog;
        // gas mass flux and continuity residual (iter.f:597-771)
        flux[0] = mflux(0, rgp);
        dg = rgp - rgpn_c + dti * diverg(flux[0]);
        bool done = loop == P.inmax;
        if (fabs(dg) > conv || fabs(dg) >= fabs(dgorig)) {
            if (nit == 1 && loop == 1) dgorig = dg;
            d3 = dg;
        } else if (fabs(dg) <= conv) {
            done = true;
        }
        if (live && done) {
            // the cell's final values: face mass fluxes (every face, as
            // calc_*_mass_flux writes them), velocities, cell state
            double *sfa = dir == 0 ? F.rsfe : (dir == 1 ? F.rsfn : F.rsft);
            gfa[fcell] = flux[0];
#pragma unroll
            for (int is = 1; is <= ns; ++is) sfa[(size_t)(is - 1) * n + fcell] = flux[is];
            if (solved) {
                gvel[fcell] = vel[0];
#pragma unroll
                for (int l = 2; l <= nph; ++l) svel[(l - 2) * n + fcell] = vel[l - 1];
            }
            mark_dirty(dirty, rawnb);
            if (q == 0) {
                F.p[c] = p; F.rog[c] = rog; F.rgp[c] = rgp; F.ep[c] = ep;
#pragma unroll
                for (int is = 1; is <= ns; ++is) F.rlk[(is - 1) * n + c] = rlk[is - 1];
                F.abeta[c] = abeta;
                mark_dirty(dirty, c);
                if (SPLIT && nit > 1 && (loop == 1) != ((e & ENTRY_LONG) != 0)) {
                    unsigned *const w = expect_long(P, dirty) + (c >> 5);
                    if (loop == 1) atomicOr(w, 1u << (c & 31));
                    else atomicAnd(w, ~(1u << (c & 31)));
                }
            }
            live = false;
        }
        if (!__any_sync(full, live)) break;
    }
}

// the inner loop of the worklist's nwork cells (outer sweep nit, 1-based) by
// the warps warp, warp + nwarps, ... of the launch, cpw <= teams per warp
// cells at a time; every lane of a warp makes the call.  RO as in ldro.
// SPLIT: the first nlong entries from the list's front are the expected long
// ones, the others stand backwards from entry last; no warp holds both, so
// that a warp of short cells ends after one iteration (a warp of five mixed
// ones hardly ever does).  Four steps of 128 x 128 x 96 with four phases 72.0
// -> 69.3 ms; three of its hills with six 95.8 -> 90.9; four of 256 x 256 x
// 192 432 -> 424, with every long cell first 443.
template <int NP, int D, bool RO, bool SPLIT = false>
__device__ __forceinline__ void inner_team_run(const Prm &P, const Fld &F, double dt, int nit, const int *list,
                                               int nwork, unsigned *dirty, int warp, int nwarps, int cpw, int nlong = 0,
                                               int last = 0) {
    constexpr int T = D == 3 ? 6 : 4;    // lanes per cell
    constexpr int TPW = 32 / T;          // teams per warp (3D: 5, lanes 30 and 31 own no face)
    const int lane = threadIdx.x & 31, tw = lane / T;
    const int q = lane - tw * T, tb = tw * T;
    extern __shared__ __align__(16) double inner_smem[];
    // every KS threads have columns of their own: [FaceK rows][KS], [3 NC][KS]
    double *const kcols = inner_smem + threadIdx.x / KS * (inner_smem_bytes<NP>() / sizeof(double));
    double *const dcols = kcols + inner_face_rows<NP>() * KS;
    if constexpr (SPLIT) {
        if (nwork <= nwarps) {  // a cell per warp: nothing to keep apart
            if (warp < nwork)
                inner_team_cell<NP, D, RO, false>(P, F, dt, nit, list[warp < nlong ? warp : last - (warp - nlong)],
                                                  tw == 0, dirty, q, tb, kcols, dcols);
            return;
        }
        // a unit is a warp's cells.  In a few rounds every warp takes long and
        // short ones in turn, those past the last long unit short ones first.
        // In many rounds what counts is that the cells at work at one time are
        // near each other in the mesh: long and short units in one sequence,
        // (u * rate) >> 32 of its first u long.  Four steps with the line at
        // eight rounds, at three, in turns throughout and in one sequence
        // throughout: 128 x 128 x 96 67.4 / 68.4 / 67.4 / 68.5 ms, its hills
        // with six phases 120.3 / 120.8 / 120.1 / 123.7, 256 x 256 x 192 405.4
        // / 404.7 / 407.7 / 403.4.
        const int nshort = nwork - nlong, ulong = (nlong + cpw - 1) / cpw, units = ulong + (nshort + cpw - 1) / cpw;
        const bool many = units > 8 * nwarps;
        const unsigned long long rate = many ? (((unsigned long long)ulong << 32) + units - 1) / units : 0;
        int l = warp, s = warp - ulong % nwarps;
        if (s < 0) s += nwarps;
        bool turn = false;
        for (int u = warp; many ? u < units : l < ulong || s < units - ulong; u += nwarps) {
            bool sh;
            int x;
            if (many) {
                const int l0 = (int)(u * rate >> 32);
                sh = (int)((u + 1) * rate >> 32) == l0;
                x = sh ? u - l0 : l0;
            } else {
                sh = l >= ulong || (turn && s < units - ulong);
                x = sh ? s : l;
                if (sh) s += nwarps;
                else l += nwarps;
                turn = !sh;
            }
            const int w0 = x * cpw, m = sh ? nshort : nlong;
            const bool live = tw < TPW && tw < cpw && w0 + tw < m;
            const int at = live ? w0 + tw : w0;
            inner_team_cell<NP, D, RO, true>(P, F, dt, nit, list[sh ? last - at : at], live, dirty, q, tb, kcols, dcols);
        }
    } else {
        for (int w0 = warp * cpw; w0 < nwork; w0 += nwarps * cpw) {
            const bool live = tw < TPW && tw < cpw && w0 + tw < nwork;
            inner_team_cell<NP, D, RO, false>(P, F, dt, nit, list[live ? w0 + tw : w0], live, dirty, q, tb, kcols, dcols);
        }
    }
}

// cells per warp of a worklist of nwork cells: while the list leaves warps
// idle each cell gets a warp of its own as far as they reach, since teams of
// one warp share its issue slots and wait for the slowest.  nwarps: the warps
// the launch may count on (one when other launches fill the device, as the
// other members of a batch do: 24 members with their cells spread out ran
// 5 % slower than packed)
template <int D>
__device__ __forceinline__ int cells_per_warp(int nwork, int nwarps) {
    constexpr int TPW = 32 / (D == 3 ? 6 : 4);
    return min(TPW, max(1, (nwork + nwarps - 1) / nwarps));
}

template <int NP, int D>
__global__ void __launch_bounds__(128, PDAC_INNER_MINB(NP)) k_inner_team(Prm P, Fld F, double dt, const int *nitp, const int *list,
                                                                     const int *count, unsigned *dirty, int spread) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int nwork = *count;
    inner_team_run<NP, D, true>(P, F, dt, *nitp, list, nwork, dirty, warp, nwarps,
                                cells_per_warp<D>(nwork, min(nwarps, spread)));
}

// Residual test of one colour phase (iter.f:241-319).
// The active set is one bit per cell: the test of a cell reads only its own
// p/rog/rgp and the mass fluxes of its faces, which change only when the
// cell or a face neighbour runs the inner loop; such a run sets the bits of
// those cells (mark_dirty).  A converged test rewrites the cell's volume
// fractions (calc_eps, from the same fluxes and rgp = ep rog): if that
// changes rgp, the next test computes a different residual, so the cell
// keeps its bit; otherwise a clean cell would recompute exactly the values
// it holds, and it is not tested.  cmask holds, per colour, the bits of the
// colour's fluid cells in the same words (k_colour_masks, set up once): a
// word's candidates are its active bits under the mask, and the bits that
// runs set on non-fluid neighbours are never looked at.  A fourth mask holds
// the plain cells (worklist entries above): flag 1 like all their face
// neighbours, no wall two cells away and none of those beyond the frame.
__global__ void k_colour_masks(Prm P, unsigned *cmask) {
    const unsigned nwords = ((unsigned)P.ncell + 31u) / 32u;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nwords) return;
    unsigned m[4] = {0u, 0u, 0u, 0u};
    for (int b = 0; b < 32; ++b) {
        const int c = (int)(32u * t) + b;
        if (c >= P.ncell) break;
        if (!(P.flag[c] & 1)) continue;
        const int i = c % P.nx + 1, r = c / P.nx, j = r % P.ny + 1, k = r / P.ny + 1;
        m[(i + j + k) % 3] |= 1u << b;
        auto axis = [&](int ii, int nax, int stride) {
            return ii >= 3 && ii <= nax - 2 && P.flag[c - stride] == FLUID && P.flag[c + stride] == FLUID &&
                   !is_wallf(P.flag[c - 2 * stride]) && !is_wallf(P.flag[c + 2 * stride]);
        };
        if (P.flag[c] == FLUID && axis(i, P.nx, 1) && axis(k, P.nz, P.nx * P.ny) && (!P.d3 || axis(j, P.ny, P.nx)))
            m[3] |= 1u << b;
    }
    for (int q = 0; q < 4; ++q) cmask[(size_t)q * nwords + t] = m[q];
}

// the residual test of cell c (iter.f:241-319): a converged cell updates its
// volume fractions and rgp (keeping its active-set bit if rgp changed);
// returns true for an unconverged cell, which goes to the inner loop
// EAGER (2D, a known phase count) asks for what a converged cell needs
// together with its residual: one trip to L2 instead of two, for more traffic
template <int NP, int D, bool EAGER>
__device__ __forceinline__ bool test_cell(const Prm &P, const Fld &F, double dt, int c, unsigned *dirty) {
    if constexpr (EAGER && D == 2 && NP > 0) {
        constexpr int ns = NP - 1;
        const int i = c % P.nx + 1, k = c / P.nx + 1;
        const int cw = at2(P, max(i - 1, 1), k), cb = at2(P, i, max(k - 1, 1));
        const CellFaces b = cell_faces(P, c);
        double fe[ns], fw[ns], ft[ns], fb[ns], ln[ns], sk[ns];
#pragma unroll
        for (int is = 1; is <= ns; ++is) {
            fe[is - 1] = SOL(F.rsfe, c, is); fw[is - 1] = SOL(F.rsfe, cw, is);
            ft[is - 1] = SOL(F.rsft, c, is); fb[is - 1] = SOL(F.rsft, cb, is);
            ln[is - 1] = SOL(F.rlkn, c, is); sk[is - 1] = SOL(F.sink, c, is);
        }
        const double old = F.rgp[c], rog = F.rog[c], conv = F.conv[c];
        const double resx = (b.e * F.rgfe[c] - b.w * F.rgfe[cw]) * P.indx[i] * P.inr[i];
        const double resz = (b.t * F.rgft[c] - b.b * F.rgft[cb]) * P.indz[k];
        const double dg = old - F.rgpn[c] + dt * b.ivf * (resx + 0.0 + resz);
        if (!(fabs(dg) <= conv)) return true;
        double rls = 0;
#pragma unroll
        for (int is = 1; is <= ns; ++is) {
            const double rx = (b.e * fe[is - 1] - b.w * fw[is - 1]) * P.indx[i] * P.inr[i];
            const double rz = (b.t * ft[is - 1] - b.b * fb[is - 1]) * P.indz[k];
            double t = ln[is - 1] - dt * b.ivf * (rx + 0.0 + rz);
            t = t + dt * b.ivf * sk[is - 1];
            const double v = fmax(0.0, t);
            SOL(F.rlk, c, is) = v;
            rls = rls + v * P.inrl[is];
        }
        const double ep = 1.0 - rls, rgp = ep * rog;
        if (rls > 1.0) atomicAdd(&F.counters[2], 1);
        F.ep[c] = ep;
        F.rgp[c] = rgp;
        if (__double_as_longlong(rgp) != __double_as_longlong(old)) mark_dirty(dirty, c);
        return false;
    }
    double dg;
    if (D == 3) {
        int i, j, k;
        ijk_of(P, c, i, j, k);
        Raw3 R;
        raw3(P, i, j, k, R);
        dg = calc_res_3d(P, F, R, i, j, k, dt);
        if (fabs(dg) <= F.conv[c]) calc_eps_3d<NP>(P, F, R, i, j, k, dt);
    } else {
        int i = c % P.nx + 1, k = c / P.nx + 1;
        Raw2 R;
        raw2(P, i, k, R);
        dg = calc_res_2d(P, F, R, i, k, dt);
        if (fabs(dg) <= F.conv[c]) calc_eps_2d(P, F, R, i, k, dt);
    }
    if (fabs(dg) <= F.conv[c]) {
        const double old = F.rgp[c];
        F.rgp[c] = F.ep[c] * F.rog[c];
        if (__double_as_longlong(F.rgp[c]) != __double_as_longlong(old)) mark_dirty(dirty, c);
        return false;
    }
    return true;
}

// One colour's residual tests by the warps warp, warp + nwarps, ... of a
// launch: each takes 32 words of the active set at a time, moves their
// candidates (clearing their bits) to its list in shared memory, tests them
// 32 at a time and appends the unconverged ones to the worklist.  The active
// cells sit close together (the plume's front), so consecutive words go to
// different warps: word by word while one round covers the mesh, else in
// groups of eight (one 32-byte sector).  slist: SCAN_LIST ints per warp.
// Collecting and testing in one pass took the two launches' fixed cost
// (about 12 us) down to one's.

// one warp's round: lane's word t (of words) of the active set under its
// colour mask, its candidates tested; put(um, lane, u, e) takes the unconverged
// ones (um: the ballot of u).  Returns the number tested.
template <int NP, int D, bool EAGER, class PUT>
__device__ __forceinline__ int scan_round(const Prm &P, const Fld &F, double dt, const unsigned *cmask,
                                          const unsigned *plain, unsigned *dirty, unsigned t, unsigned nwords,
                                          int *slist, PUT put, const unsigned *expect = nullptr) {
    constexpr unsigned full = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    unsigned w = 0, pl = 0, lg = 0;
    if (t < nwords) {
        if (expect) lg = __ldcg(expect + t);
        w = __ldcg(dirty + t) & __ldg(cmask + t);
        pl = __ldg(plain + t);
        if (w) atomicAnd(dirty + t, ~w);
    }
    int incl = __popc(w);
    const int mine = incl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= (unsigned)o) incl += v;
    }
    const int total = __shfl_sync(full, incl, 31);
    if (total == 0) return 0;
    for (int off = incl - mine; w; w &= w - 1u) {
        const int b = __ffs(w) - 1;
        slist[off++] = (int)(32u * t + (unsigned)b | (pl >> b & 1u) << 31 | (lg >> b & 1u) << 30);
    }
    __syncwarp();
    for (int base = 0; base < total; base += 32) {
        const int idx = base + (int)lane;
        int e = 0;
        bool u = false;
        if (idx < total) {
            e = slist[idx];
            u = test_cell<NP, D, EAGER>(P, F, dt, entry_cell(e), dirty);
        }
        const unsigned um = __ballot_sync(full, u);
        if (um) put(um, lane, u, e);
    }
    __syncwarp();  // the list is read before the next round overwrites it
    return total;
}

// a phase's test by all warps of a grid: put as scan_round's; returns the
// number of cells this warp tested
template <int NP, int D, class PUT>
__device__ __forceinline__ int scan_phase(const Prm &P, const Fld &F, double dt, const unsigned *cmask,
                                          const unsigned *plain, unsigned *dirty, unsigned warp, unsigned nwarps,
                                          int *slist, PUT put, const unsigned *expect = nullptr) {
    const unsigned lane = threadIdx.x & 31u, nwords = ((unsigned)P.ncell + 31u) / 32u;
    const unsigned gs = nwords <= 32u * nwarps ? 1u : 8u, gpi = 32u / gs;  // words per group, groups per round
    int ntest = 0;
    for (unsigned g0 = 0; (size_t)g0 * nwarps * gs < nwords; g0 += gpi) {
        const unsigned t = ((g0 + lane / gs) * nwarps + warp) * gs + lane % gs;
        ntest += scan_round<NP, D, false>(P, F, dt, cmask, plain, dirty, t, nwords, slist, put, expect);
    }
    return ntest;
}

template <int NP, int D>
__global__ void __launch_bounds__(TPB_RESID) k_resid_scan(Prm P, Fld F, double dt, const unsigned *cmask,
                                                          const unsigned *plain, unsigned *dirty, int *work, int *count) {
    __shared__ int slist[TPB_RESID / 32][SCAN_LIST];
    const unsigned warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int ntest = scan_phase<NP, D>(P, F, dt, cmask, plain, dirty, warp, nwarps, slist[threadIdx.x >> 5],
                                        [&](unsigned um, unsigned ln, bool u, int e) {
                                            int at = 0;
                                            if (ln == 0) at = atomicAdd(count, __popc(um));
                                            at = __shfl_sync(0xffffffffu, at, 0);
                                            if (u) work[at + __popc(um & ((1u << ln) - 1u))] = e;
                                        });
    if ((threadIdx.x & 31u) == 0 && ntest) atomicAdd(count + 3, ntest);
}

// The whole outer sweep loop of iter (iter.f:204-410) in one launch whose
// blocks are all resident: the colour phases' residual tests and inner loops
// follow each other across barriers instead of launches.
// Every thread takes every barrier the same number of times: the loop ends
// on counters that all threads read after the same barrier.
struct SweepWork {
    int *wcount;      // on return: [col] worklist length of the last sweep
    // two sets of three worklist lengths, for odd and even sweeps: the
    // expected long cells in the low half, the others in the high half
    unsigned long long *counts;
    int *work;        // worklists, colour col at work + col * wstride
    unsigned *dirty;  // active set, one bit per cell
    const unsigned *cmask;  // the three colour masks and the plain mask
    int *nit;         // the sweep count on return, as the graph's k_sweep_check leaves it
    long wstride;     // ints per colour's worklist
};

// after a sweep's last barrier: its worklist lengths; true when the loop ends
__device__ __forceinline__ bool sweep_ends(const SweepWork &W, const unsigned long long *cnt, int nit, int maxout) {
    auto length = [](unsigned long long v) { return (int)(v & 0xffffffffu) + (int)(v >> 32); };
    const int n0 = length(__ldcg(cnt)), n1 = length(__ldcg(cnt + 1)), n2 = length(__ldcg(cnt + 2));
    const bool conv = (long)n0 + n1 + n2 == 0;
    if (!conv && nit < maxout) return false;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        W.wcount[0] = n0;
        W.wcount[1] = n1;
        W.wcount[2] = n2;
        *W.nit = conv ? nit : maxout + 1;
    }
    return true;
}

// on a cooperative grid: the unconverged cells of a phase go to one worklist,
// from which all warps take theirs, a grid-wide barrier after either half
template <int NP, int D>
__global__ void __launch_bounds__(KS, PDAC_INNER_MINB(NP)) k_sweep_grid(Prm P, Fld F, double dt, SweepWork W, int maxout) {
    auto barrier = [] { cooperative_groups::this_grid().sync(); };
    extern __shared__ __align__(16) double inner_smem[];
    const int wid = threadIdx.x >> 5, warp = blockIdx.x * (KS / 32) + wid, nwarps = gridDim.x * (KS / 32);
    const unsigned nwords = ((unsigned)P.ncell + 31u) / 32u;
    // the scan's list and the inner loop's columns are never live together
    int *const slist = reinterpret_cast<int *>(inner_smem) + wid * SCAN_LIST;
    if (blockIdx.x == 0 && threadIdx.x < 6) W.counts[threadIdx.x] = 0;
    barrier();
    for (int nit = 1;; ++nit) {
        unsigned long long *const cnt = W.counts + 3 * (nit & 1), *const other = W.counts + 3 * (~nit & 1);
        for (int col = 0; col < 3; ++col) {
            int *const work = W.work + col * W.wstride;
            const int last = (int)W.wstride - 1;
            // after the last sweep the list is read from its front
            const bool all_long = nit == maxout;
            scan_phase<NP, D>(P, F, dt, W.cmask + (size_t)col * nwords, W.cmask + (size_t)3 * nwords, W.dirty, warp,
                              nwarps, slist,
                              [&](unsigned um, unsigned ln, bool u, int e) {
                                  const unsigned lm = __ballot_sync(0xffffffffu, u && (all_long || (e & ENTRY_LONG))), sm = um & ~lm;
                                  unsigned long long at = 0;
                                  if (ln == 0)
                                      at = atomicAdd(cnt + col, (unsigned long long)__popc(sm) << 32 | (unsigned)__popc(lm));
                                  at = __shfl_sync(0xffffffffu, at, 0);
                                  const unsigned before = (1u << ln) - 1u;
                                  if (lm >> ln & 1u) work[(int)(at & 0xffffffffu) + __popc(lm & before)] = e;
                                  else if (u) work[last - (int)(at >> 32) - __popc(sm & before)] = e;
                              },
                              expect_long(P, W.dirty));
            __syncwarp();
            barrier();
            const unsigned long long lens = __ldcg(cnt + col);
            const int nlong = (int)(lens & 0xffffffffu), nwork = nlong + (int)(lens >> 32);
            // the next sweep's lengths: last read before this sweep's first barrier
            if (col == 1 && blockIdx.x == 0 && threadIdx.x < 3) other[threadIdx.x] = 0;
            if (nwork) {
                constexpr int TPW = 32 / (D == 3 ? 6 : 4);
                int cpw = cells_per_warp<D>(nwork, nwarps);  // a unit per warp, where they go round
                while (cpw < TPW && (nlong + cpw - 1) / cpw + (nwork - nlong + cpw - 1) / cpw > nwarps) ++cpw;
                inner_team_run<NP, D, false, true>(P, F, dt, nit, work, nwork, W.dirty, warp, nwarps, cpw, nlong, last);
            }
            __syncwarp();
            barrier();
        }
        if (sweep_ends(W, cnt, nit, maxout)) return;
    }
}

// On one thread-block cluster, for small 2D meshes, whose phases hold a few
// hundred cells: what bounds a phase is the number of dependent trips to L2
// on its way (0.3 to 0.5 us each; the inner loop itself is one or three
// iterations of 0.75 us).  So a block keeps the unconverged cells of its own
// words in shared memory -- no global list, count or second barrier between
// test and inner loop -- and the words of a neighbourhood are dealt out to
// different blocks: of every CLUSTER consecutive words each block has one,
// turned by 7 from one group to the next, so that a front running down the
// columns of a mesh of any width meets all blocks.  The hardware schedules a
// cluster's blocks together, so any number of such launches may share the
// device.  Ten steps of 128 x 192: 35.0 ms with a common worklist, 32.2 here.
// Eight warps a block hide one another's trips where a phase has more cells
// than the cluster has warps: five steps of 251 x 383, 38.0 ms with four
// (36.3 with the common worklist), 30.8 with eight; 128 x 192 the same.
constexpr int CLUSTER = 16, KC = 256;  // blocks; their threads, each with a word of the active set at most
template <int NP>
__host__ __device__ constexpr size_t cluster_smem_bytes() {
    return sweep_smem_bytes<NP>(KC) + KC * WORD_CELLS * sizeof(int);
}
template <int NP>
__global__ void __launch_bounds__(KC, 1) k_sweep_cluster(Prm P, Fld F, double dt, SweepWork W, int maxout) {
    extern __shared__ __align__(16) double inner_smem[];
    __shared__ int nmine, base;
    int *const mine = reinterpret_cast<int *>(reinterpret_cast<char *>(inner_smem) + sweep_smem_bytes<NP>(KC));
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const unsigned nwords = ((unsigned)P.ncell + 31u) / 32u, b = blockIdx.x;
    int *const slist = reinterpret_cast<int *>(inner_smem) + wid * SCAN_LIST;
    auto barrier = [] {
        __syncwarp();
        cooperative_groups::this_cluster().sync();
    };
    if (b == 0 && threadIdx.x < 6) W.counts[threadIdx.x] = 0;
    if (threadIdx.x == 0) nmine = 0;
    barrier();
    for (int nit = 1;; ++nit) {
        unsigned long long *const cnt = W.counts + 3 * (nit & 1), *const other = W.counts + 3 * (~nit & 1);
        for (int col = 0; col < 3; ++col) {
            const unsigned g = wid + KC / 32 * lane;  // this thread's group of CLUSTER words
            scan_round<NP, 2, true>(P, F, dt, W.cmask + (size_t)col * nwords, W.cmask + (size_t)3 * nwords, W.dirty,
                                    g * CLUSTER + ((b + 7u * g) & (CLUSTER - 1u)), nwords, slist,
                                    [&](unsigned um, unsigned ln, bool u, int e) {
                                        int at = 0;
                                        if (ln == 0) at = atomicAdd(&nmine, __popc(um));
                                        at = __shfl_sync(0xffffffffu, at, 0);
                                        if (u) mine[at + __popc(um & ((1u << ln) - 1u))] = e;
                                    });
            __syncthreads();
            const int nwork = nmine;
            if (threadIdx.x == 0 && nwork) base = (int)atomicAdd(cnt + col, (unsigned long long)nwork);
            if (nit == maxout && nwork) {  // the cells a loop without convergence reports
                __syncthreads();
                for (int q = threadIdx.x; q < nwork; q += KC) W.work[col * W.wstride + base + q] = mine[q];
            }
            // the next sweep's lengths: last read before this sweep's first barrier
            if (col == 1 && b == 0 && threadIdx.x < 3) other[threadIdx.x] = 0;
            if (nwork)
                inner_team_run<NP, 2, false>(P, F, dt, nit, mine, nwork, W.dirty, wid, KC / 32,
                                             cells_per_warp<2>(nwork, KC / 32));
            __syncthreads();  // the list and its length are done with
            if (threadIdx.x == 0) nmine = 0;
            barrier();
        }
        if (sweep_ends(W, cnt, nit, maxout)) return;
    }
}

// End of one outer sweep on the device (iter.f:388-410): with no unconverged
// cell left, or after maxout sweeps, the sweep loop stops; otherwise the
// sweep number advances.  *nit ends as the host loop's nit (maxout + 1 when
// the sweeps did not converge).
__global__ void k_sweep_check(const int *wcount, int *nit, int maxout, cudaGraphConditionalHandle loop) {
    long unconverged = (long)wcount[0] + wcount[1] + wcount[2];
    if (unconverged == 0) { cudaGraphSetConditional(loop, 0); return; }
    if (*nit >= maxout) { *nit = maxout + 1; cudaGraphSetConditional(loop, 0); return; }
    *nit += 1;
    cudaGraphSetConditional(loop, 1);
}

}  // namespace pdac
