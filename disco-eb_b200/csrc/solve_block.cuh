// The adaptive solve of one k-mode on a block of warps (device only).
//
// Same discrete solve as solve_mode / rodas5_step (stepper.cuh), operation for operation: every
// row, chain element, functional and controller value is the same expression on the same
// operands, so the accepted steps and the states are bit for bit those of the one-warp form (the
// step control amplifies a last-bit difference into a different accept decision in about one mode
// of four at rtol 1e-5, so anything less would change results).  What changes is where each
// piece runs and when:
//
//   warp 0      "special"  the special rows and metric functionals of every stage, the controller,
//                          the output stage; one lane per special row for the rest of a stage
//   warp 1      "chains"   the factorisation and the substitutions, a lane per (chain, right-hand
//                          side): A^{-1} U and stage 0 are solved together
//   warps 2..   "rows"     the hierarchy rows, one row per thread (as many warps as that takes)
//   last but 1  "scale"    the scale factor obeys a scalar equation of its own (row 0 of W is
//                          1 x 1), so its eight stages, and with them every stage's table lookups,
//                          run ahead of the other rows instead of on their critical path
//   last        "prep"     finishes the stage backgrounds the scale warp looked up and, after the
//                          last one, prepares the next step's point (dual background, special rows
//                          of S and U, functionals G and F1) on the assumption that the step is
//                          accepted; a rejected step keeps the prepared point of its start (same
//                          inputs, so the same values) and its dual right-hand side.
//
// What bounds it: dependent latency.  One warp per mode spent ~190 k cycles per step attempt
// (96 us), nearly all of it in code that one warp runs serially while its other lanes idle (15
// special rows, 5 table lookups, 8 chains); the warps here overlap those.
//
// Warps meet at hardware barriers only (bar.sync / bar.arrive): 0 whole block, 1 special + rows,
// 2 scale + prep, 3..9 stage 1..7's background (prep arrives, special + rows wait), 10 the stage-0
// value of the scale-factor chain (scale arrives), 11 special + chains + rows.  Every role executes
// the same barriers in the same order in every step, whatever the step's outcome.
#pragma once

#include "stepper.cuh"

#if defined(__CUDACC__)

namespace dscb {
namespace blk {

// warps of a mode: special, chains, rows, scale, prep
inline __host__ __device__ int row_warps(const Dims& D) { return (n_hier_rows(D) + 31) / 32; }
inline __host__ __device__ int block_threads(const Dims& D) { return 32 * (row_warps(D) + 4); }

// (bar.sync and bar.arrive count whole warps: the lanes meet first)
__device__ __forceinline__ void bar_sync(int id, int count)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count)
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Where a fused multiply-add can form in more than one place of an expression the compiler's choice
// depends on the code around it, and these few choices differ between this kernel and the one-warp
// kernels when both are written alike.  They are pinned here to the one-warp kernels' (each found by
// comparing single steps, bit for bit, over random states in every regime), as nvcc 12.9 compiles those:
// another compiler may choose otherwise there, and the tests that compare the two forms then tell.
struct Rounding {
    // 3 (a'/a)^2, from the massive-neutrino density
    static __device__ __forceinline__ double friedmann(const DiscoebCosmo& P, double grhom, double Omegam, double OmegaDE,
                                                       double ia, double ia2, double a2, double rho_Q, double rhonu,
                                                       bool fuse_de)
    {
        const double X = __fma_rn(P.grhor, __fma_rn(P.Nmnu, rhonu, P.Neff), P.grhog);
        const double W = __dmul_rn(__dmul_rn(grhom, OmegaDE), rho_Q);
        const double s = __fma_rn(__dmul_rn(grhom, Omegam), ia, __dmul_rn(X, ia2));
        return __fma_rn(grhom, P.Omegak, fuse_de ? __fma_rn(W, a2, s) : __dadd_rn(s, __dmul_rn(W, a2)));
    }
    __device__ __forceinline__ double operator()(const DiscoebCosmo& P, const Par<double>& par, const Bg<double>& b,
                                                 const BgTables<double>& tb) const
    {
        return friedmann(P, par.grhom, par.Omegam, par.OmegaDE, b.ia, b.ia2, b.a2, b.rho_Q, tb.rhonu, true);
    }
    __device__ __forceinline__ Dual operator()(const DiscoebCosmo& P, const Par<Dual>& par, const Bg<Dual>& b,
                                               const BgTables<Dual>& tb) const
    {
        return Dual(friedmann(P, par.grhom.v, par.Omegam.v, par.OmegaDE.v, b.ia.v, b.ia2.v, b.a2.v, b.rho_Q.v, tb.rhonu.v,
                              false),
                    Friedmann()(P, par, b, tb).d);
    }
    // the dark-energy sound speed's ca2 = w - w'/(3 (1 + w) a'/a)
    static __device__ __forceinline__ double ca2(double wa, double aH, double a, double w_Q, double inv_opw)
    {
        return __fma_rn(-__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(-wa, aH), a), 1.0 / 3.0), inv_opw), rcp(aH), w_Q);
    }
    static __device__ __forceinline__ Dual product(const Dual& x, const Dual& y)  // rho_Q a^2 of the dual special rows
    {
        return Dual(__dmul_rn(x.v, y.v), __fma_rn(x.v, y.d, __dmul_rn(x.d, y.v)));
    }
    // theta_gamma under radiation streaming and the bracket inside it
    static __device__ __forceinline__ double theta(double H, double fac, double Y) { return __fma_rn(fac, Y, -0.5 * H); }
    static __device__ __forceinline__ double inner(double a, double x, double b, double y, double c, double z)
    {
        return __dadd_rn(__dmul_rn(c, z), __fma_rn(b, y, __dmul_rn(a, x)));
    }
    static __device__ __forceinline__ double product(double x, double y) { return x * y; }
    static __device__ __forceinline__ double rsa_theta(double H, double fac, double Y) { return theta(H, fac, Y); }
    static __device__ __forceinline__ Dual rsa_theta(const Dual& H, const Dual& fac, const Dual& Y)
    {
        return Dual(theta(H.v, fac.v, Y.v), (-0.5 * H + fac * Y).d);
    }
    static __device__ __forceinline__ double rsa_inner(double a, double x, double b, double y, double c, double z)
    {
        return inner(a, x, b, y, c, z);
    }
    static __device__ __forceinline__ Dual rsa_inner(const Dual& a, double x, const Dual& b, double y, double c, double z)
    {
        return Dual(inner(a.v, x, b.v, y, c, z), (a * x + b * y + c * z).d);
    }
    // -band entry (baryon velocity, baryon density) under radiation streaming
    static __device__ __forceinline__ double rsa_baryon(const Bg<double>& b, double k)
    {
        const double k2 = k * k, sk2 = k2 > 1e-30 ? k2 : 1e-30;
        return __fma_rn(__dmul_rn(b.po, b.rsa_fac), __dmul_rn(b.cs2, sk2), __dmul_rn(k2, b.cs2));
    }
    // (8/15) (theta + k^2 alpha) - 0.6 k F_3: the l = 2 rows of photons and massless neutrinos
    static __device__ __forceinline__ double alpha(double hprime, double etaprime, double k2)
    {
        return __dmul_rn(__fma_rn(6.0, etaprime, hprime), 0.5 / k2);
    }
    static __device__ __forceinline__ double shear_row(double k, double yl3, double theta, double k2, double alpha)
    {
        return __fma_rn(8.0 / 15.0, __dadd_rn(theta, __dmul_rn(k2, alpha)), -__dmul_rn(0.6 * k, yl3));
    }
    static __device__ __forceinline__ double thomson(double f, double opac, double shear, double polter)
    {
        return __fma_rn(-opac, __fma_rn(-0.1, polter, shear), f);
    }
    // the two rows in sp[9] and sp[12], from the state through Y
    template <class YF>
    static __device__ __forceinline__ void shear_rows(const Dims& D, const Bg<double>& b, double k, double tau, YF Y,
                                                      double hprime, double etaprime, double polter, double& sp9,
                                                      double& sp12)
    {
        if (b.rsa) return;
        const double k2 = k * k, al = alpha(hprime, etaprime, k2);
        sp9 = thomson(shear_row(k, Y(10), Y(8), k2, al), b.opac, Y(9), polter);
        sp12 = b.ufa ? ufa_shear(tau, b.itau, Y(D.idxr + 2), Y(D.idxr + 1), hprime)
                     : shear_row(k, Y(D.idxr + 3), Y(D.idxr + 1), k2, al);
    }
    // massless-neutrino shear under the fluid closure
    static __device__ __forceinline__ double ufa_shear(double tau, double itau, double yr2, double thr, double hprime)
    {
        return __fma_rn(-1.5 * (tau > 1e-30 ? itau : 1e30), yr2, __dmul_rn(4.0 / 15.0, __fma_rn(0.5, hprime, thr)));
    }
};

// what a step needs of its start point (t, y_0, regime) besides the state
struct Point {
    Bg<Dual> bd;               // background with d/da
    Bg<double> b;              // its value part
    Dual iv[DISCOEB_MAX_NQ], v[DISCOEB_MAX_NQ];  // 1/v and v of the momentum bins, with d/da
    double vf[DISCOEB_MAX_NQ]; // v of the momentum bins
    // special rows of S and U: lower, main and upper diagonal, the three U columns
    double row[15][6];
    double s68, s86, etac, f1u[3];  // S's entries (6, 8), (8, 6); row 6's eta coefficient; F1 U
    double t, it2;                  // time and its inverse square
    int regime;                     // what `row` was laid out for (-1: nothing)
    double Gs[3 * kMaxSlots], F1s[kMaxSlots];
};
struct Stage {
    Bg<double> b;
    double iv[DISCOEB_MAX_NQ], v[DISCOEB_MAX_NQ];
    double x0;  // K_s[0]
    BgTables<double> tb;
    double a, ts;
};
// Who may read what, and when.  Warp 0's controller writes the fields marked (c) between barrier 1 at
// the end of one attempt and barrier 0 at the start of the next.  Of the other warps it has then met
// only special + rows (barrier 1) since the attempt's last stage, so these read them anywhere between
// the two; the chains read theirs before their last barrier 11, the scale warp before it arrives at
// barrier 10 and the prep warp before its last arrival at barriers 3..9.  What the scale or prep warp
// needs later, while it prepares the next point, it keeps in registers.
struct Ctl {
    double t, h, tnext;               // (c)
    int regime, go, fresh, accepted;  // (c); fresh: the point differs from the previous attempt's
    int nbad_cand, nbad_start, fac_ok;  // (c), then counted by the attempt's warps
    double g[3], gd[3];       // metric functionals of the stage (and d/da at the point)
    double sp[16];            // special rows of the stage's right-hand side
    double dlq[DISCOEB_MAX_NQ];
    double cmat[9], gz0[4];   // C = I - G Z, G and F1 applied to stage 0's chains
    double y0_next;           // (c) row 0 of an accepted candidate
    double pw[2];             // the controller's powers of the two previous errors, from the prep warp
    double e2, e3;            // (c) those errors (inverse) for the prep warp
    double au2, al2;          // W's two entries outside the tridiagonal chains: (6, 8) and (8, 6)
    double cih[8][8], hd[8];  // C_sj / h, h d_s
};
struct Shared {
    Point pt[2];
    Stage st[8];
    Ctl c;
};
constexpr int kSharedDoubles = (sizeof(Shared) + 7) / 8;
constexpr int kCosmo = (sizeof(DiscoebCosmo) + 7) / 8;

// positions from one element of a chain to the next: the long chains (three and one per momentum bin),
// rounded up to one of two widths
constexpr int kNarrow = 8, kWide = 20;
inline __host__ __device__ int chain_stride(const Dims& D) { return 3 + D.nq <= kNarrow ? kNarrow : kWide; }
// Positions per chain: the longest chain, rounded up to what the substitutions are written for.  Narrow
// chains up to kLong take one of two lengths that keep their intermediate results in registers
// (solve_tri_s); longer ones go by fours (solve_tri_n).  Two lengths, because a body for every four up to
// 24 makes all states slower through their code (512 modes with tangents, 143 rows 141 -> 152 ms, 72 rows
// 151 -> 157); rounded up to these two, chains of 4 to 8 and 13 to 16 gain over the loop (256 modes, 8
// positions 27.8 -> 25.9 ms, 16 positions 29.8 -> 26.7; tangents of 512 modes 153 -> 148, 158 -> 156).
constexpr int kShort = 12, kLong = 20;
inline __host__ __device__ int chain_steps(const Dims& D)
{
    int L = D.lmaxg;
    L = L > D.lmaxgp + 1 ? L : D.lmaxgp + 1;
    L = L > D.lmaxr + 1 ? L : D.lmaxr + 1;
    if (D.nq > 0) L = L > D.lmaxnu + 1 ? L : D.lmaxnu + 1;
    if (chain_stride(D) == kNarrow && L <= kLong) return L <= kShort ? kShort : kLong;
    return (L + 3) & ~3;
}
inline __host__ __device__ int positions_of(const Dims& D) { return chain_steps(D) * chain_stride(D) + 9; }
// doubles of shared memory of one mode:
// the state vectors and stages (13 n), the functionals and scalars, the chains (8 per position)
inline __host__ __device__ int block_mem_doubles(const Dims& D)
{
    // (the last column's look-ahead reads four elements past the positions)
    return 13 * D.n + 4 * kMaxSlots + 32 + 8 * positions_of(D) + 4 * chain_stride(D) + 2;
}
inline __host__ __device__ int smem_doubles(const Dims& D) { return kCosmo + block_mem_doubles(D) + kSharedDoubles; }
__device__ __forceinline__ ModeMem block_carve(double* base, const Dims& D)
{
    ModeMem m = carve(base, D);
    m.Gs = base + 13 * D.n;
    m.F1s = m.Gs + 3 * kMaxSlots;
    m.sc = m.F1s + kMaxSlots;
    double* chains = m.sc + 32;  // 16-byte aligned
    m.A = chains + ((reinterpret_cast<uintptr_t>(chains) & 8u) ? 1 : 0);
    m.Z = nullptr;
    return m;
}

static __device__ __noinline__ double div_call(double x, double y) { return x / y; }
static __device__ __noinline__ double pow_call(double x, double p) { return pow(x, p); }

// ---- the scale and prep warps: the scale-factor chain, stage backgrounds, next point ----

// The special rows of S and U at a point (rowc): what depends on the point is written every time,
// the constants when the regime changes.  One lane.
__device__ __forceinline__ void point_rows(const DiscoebCosmo& P, double k, double tau, Point& pt)
{
    const Bg<double>& b = pt.b;
    const double k2 = k * k, sk2 = k2 > 1e-30 ? k2 : 1e-30;
    const int regime = (b.rsa ? 1 : 0) | (b.ufa ? 2 : 0) | (b.de_frozen ? 8 : 0);
    enum { LO, DI, UP, U0, U1, U2 };
    auto& w = pt.row;
    if (regime != pt.regime) {
        for (int r = 0; r < 15; ++r)
            for (int c = 0; c < 6; ++c) w[r][c] = 0.0;
        w[2][U1] = 1.0;
        w[3][UP] = w[5][UP] = -1.0;
        w[3][U0] = w[5][U0] = -0.5;
        pt.s68 = pt.s86 = pt.etac = 0.0;
        if (!b.rsa) {
            w[7][UP] = w[10][UP] = -4.0 / 3.0;
            w[7][U0] = w[10][U0] = -2.0 / 3.0;
            w[8][LO] = w[11][LO] = 0.25 * k2;
            w[8][UP] = w[11][UP] = -0.5 * k2;
            w[9][LO] = 8.0 / 15.0;
            w[9][UP] = -0.6 * k;
            w[9][U0] = 4.0 / 15.0;
            w[9][U1] = 8.0 / 5.0;
            if (b.ufa) {
                w[12][LO] = 4.0 / 15.0;
                w[12][U0] = 2.0 / 15.0;
            } else {
                w[12][LO] = 8.0 / 15.0;
                w[12][UP] = -0.6 * k;
                w[12][U0] = 4.0 / 15.0;
                w[12][U1] = 8.0 / 5.0;
            }
        }
        pt.regime = regime;
    }
    w[4][DI] = -b.aH;
    if (b.rsa) {
        const double pf = b.po * b.rsa_fac;
        w[6][LO] = Rounding::rsa_baryon(b, k);
        w[6][DI] = __fma_rn(pf, -b.rsa_tcs - b.aH, -b.aH - b.po);
        pt.etac = pf * sk2;
        w[6][U0] = b.po * __fma_rn(-(0.5 * b.rsa_fac), b.rsa_tcs, -0.5);
    } else {
        w[6][LO] = k2 * b.cs2;
        w[6][DI] = -b.aH - b.po;
        pt.s68 = b.po;
        pt.s86 = b.opac;
        w[8][DI] = w[9][DI] = -b.opac;
        w[9][U2] = 0.1 * b.opac;
        if (b.ufa) w[12][DI] = -1.5 * (tau > 1e-30 ? b.itau : 1e30);
    }
    if (!b.de_frozen) {
        const double cs2Q = P.cs2_DE;
        w[13][DI] = -3.0 * (cs2Q - b.w_Q) * b.aH;
        w[13][UP] = __fma_rn(-(9.0 * b.opw * (cs2Q - b.ca2_Q) * b.aH * b.aH), rcp(k2), -b.opw);
        w[13][U0] = -0.5 * b.opw;
        w[14][LO] = cs2Q * b.iopw * k2;
        w[14][DI] = -(1.0 - 3.0 * cs2Q) * b.aH;
    }
}

// The functionals G and F1 on the state slots (gcol, f1col) and F1 U: lane 0 the fluids, lane q the
// momentum bins
__device__ __forceinline__ void point_functionals(const WarpTeam& tm, const DiscoebCosmo& P, const Dims& D, double k,
                                                  Point& pt)
{
    const Bg<double>& b = pt.b;
    const double k2 = k * k, sk2 = k2 > 1e-30 ? k2 : 1e-30, hE = 0.5 / k2, third = 1.0 / 3.0;
    const double Omegac = b.par.Omegam - b.par.Omegab, ih = b.iaHG, ia = b.ia, ia2 = b.ia2;
    const bool rsa = b.rsa;
    const int nq = D.nq, de = 12 + 2 * nq;
    double* g0 = pt.Gs;
    double* g1 = pt.Gs + kMaxSlots;
    double* g2 = pt.Gs + 2 * kMaxSlots;
    double* f1 = pt.F1s;
    const double fac = b.rsa_fac, cg = hE * (4.0 / 3.0) * P.grhog * ia2;
    double eH = 0.0;
    if (rsa)
        eH = __fma_rn(cg, __fma_rn(-(0.5 * fac), b.rsa_tcs, -0.5),
                      hE * (4.0 / 3.0) * P.Neff * P.grhor * ia2 * (-0.5));
    if (tm.leader()) {
        const double c = b.par.grhom * Omegac * ia, bb = b.par.grhom * b.par.Omegab * ia;
        const double eta = 2.0 * k2 * ih, gc = c * ih, gb = bb * ih;
        const double pg = P.grhog * ia2, pr = P.grhor * P.Neff * ia2;
        const double dq = b.par.grhom * b.par.OmegaDE * b.rho_Q * b.a2, gq = dq * ih;
        const double tb = hE * b.par.grhom * b.par.Omegab * ia;
        g0[0] = eta; g0[1] = gc; g0[2] = 0.0; g0[3] = gb; g0[4] = 0.0;
        g0[5] = rsa ? 0.0 : pg * ih;
        g0[6] = g0[7] = g0[8] = g0[9] = g0[11] = 0.0;
        g0[10] = rsa ? 0.0 : pr * ih;
        g0[de] = gq;
        g0[de + 1] = 0.0;
        g1[0] = rsa ? __fma_rn(eH, eta, cg * fac * sk2) : 0.0;
        g1[1] = eH * gc;
        g1[2] = hE * b.par.grhom * Omegac * ia;
        g1[3] = rsa ? __fma_rn(eH, gb, cg * fac * (b.cs2 * sk2)) : 0.0;
        g1[4] = rsa ? __fma_rn(cg * fac, -b.rsa_tcs - b.aH, tb) : tb;
        g1[5] = g1[7] = g1[8] = g1[9] = g1[10] = 0.0;
        g1[6] = rsa ? 0.0 : cg;
        g1[11] = rsa ? 0.0 : hE * (4.0 / 3.0) * P.Neff * P.grhor * ia2;
        g1[de] = eH * gq;
        g1[de + 1] = hE * b.opw * b.rho_Q * b.par.grhom * b.par.OmegaDE * b.a2;
        for (int q = 0; q < 12; ++q) g2[q] = 0.0;
        g2[de] = g2[de + 1] = 0.0;
        if (!rsa) g2[7] = g2[8] = g2[9] = 1.0;
        const double presq = (P.cs2_DE - b.ca2_Q) *
                             (3.0 * b.aH * b.opw * b.rho_Q * b.par.grhom * b.par.OmegaDE * b.a2 * rcp(k2));
        for (int q = 0; q < 12; ++q) f1[q] = 0.0;
        f1[1] = -b.a * c;
        f1[3] = -b.a * bb;
        f1[5] = -b.a * (rsa ? pg : pg + 3.0 * (pg * third));
        f1[10] = -b.a * (rsa ? pr : pr + 3.0 * (pr * third));
        f1[de] = -b.a * (dq + 3.0 * (P.cs2_DE * b.par.grhom * b.par.OmegaDE * b.rho_Q * b.a2));
        f1[de + 1] = -b.a * (3.0 * presq);
        pt.f1u[0] = pt.f1u[1] = pt.f1u[2] = 0.0;
        if (rsa) {
            const double itc = fac * (sk2 * third);
            f1[0] = -b.a * (3.0 * ((P.grhog + P.grhor * P.Neff) * ia2 * third * (-4.0)));
            f1[4] = -b.a * (3.0 * (pg * third * (4.0 * rcp(sk2)) * itc));
            const double q4 = 4.0 * b.aH * rcp(sk2);
            pt.f1u[0] = -b.a * 3.0 * (pg * third * (q4 + 2.0 * rcp(sk2) * itc) + pr * third * q4);
        }
    }
    if (tm.lane < nq) {
        const int q = tm.lane;
        const double iv = inv_vq(P, b, q), wq = P.wq[q];
        const double rho = P.grhor * P.Nmnu * wq * iv * ia2, g = rho * ih;
        pt.vf[q] = rcp(iv);
        g0[12 + q] = g;
        g1[12 + q] = eH * g;
        g2[12 + q] = g2[12 + nq + q] = 0.0;
        g0[12 + nq + q] = 0.0;
        g1[12 + nq + q] = hE * P.Nmnu * P.grhor * k * wq * ia2;
        f1[12 + q] = -b.a * (rho + 3.0 * (P.grhor * P.Nmnu * ia2 * wq * pt.vf[q] * third));
        f1[12 + nq + q] = 0.0;
        pt.iv[q] = inv_vq(P, pt.bd, q);
        pt.v[q] = rcp(pt.iv[q]);
    }
}

// The scale warp's table lookups: lane t (0..3) keeps its table's current interval, which consecutive
// stages rarely leave (bg_tables' lookup and evaluation, spline_eval_at / spline_deriv_at with the
// interval's constants formed once).
struct Interval {
    double x0, xi, xj, uinv;       // first knot and inverse spacing (uniform tables), the interval's knots
    double rh, h26, yi, yj, Si, Sj, d0, d1, d2;
    int i, n;
    bool uniform;
};
__device__ __forceinline__ void load_interval(const DiscoebSpline& s, int i, Interval& v)
{
    v.i = i;
    v.xi = DLDG(s.x + i);
    v.xj = DLDG(s.x + i + 1);
    v.yi = DLDG(s.y + i);
    v.yj = DLDG(s.y + i + 1);
    v.Si = DLDG(s.S + i);
    v.Sj = DLDG(s.S + i + 1);
    const double h = v.xj - v.xi;
    v.rh = rcp(h);
    v.h26 = div_call(__dmul_rn(h, h), 6.0);
    // slope: d0 + d1 d + d2 d^2
    v.d0 = __fma_rn(v.yj - v.yi, v.rh, -__dmul_rn(__dmul_rn(h, __fma_rn(2.0, v.Si, v.Sj)), 1.0 / 6.0));
    v.d1 = 2.0 * (v.Si * 0.5);
    v.d2 = 3.0 * ((v.Sj - v.Si) * rcp(6.0 * h));
}
__device__ __forceinline__ void init_interval(const WarpTeam& tm, const DiscoebCosmo& P, Interval& v)
{
    const DiscoebSpline& s = table_slot_spline(P, tm.lane < 4 ? tm.lane : 0);
    v.n = s.n_knots;
    v.uniform = s.uniform != 0;
    v.x0 = DLDG(s.x);
    v.uinv = v.uniform ? rcp(DLDG(s.x + 1) - v.x0) : 0.0;
    load_interval(s, v.uniform ? 0 : v.n / 2, v);
}
__device__ __forceinline__ BgTables<double> stage_tables(const WarpTeam& tm, const DiscoebCosmo& P,
                                                         const Par<double>& par, double a, Interval& v)
{
    const double loga = xlog(a);
    bool stale;
    int want = 0;
    if (v.uniform) {
        const double fi = floor((loga - v.x0) * v.uinv);
        want = !(fi >= 0.0) ? 0 : (fi > (double)(v.n - 2) ? v.n - 2 : (int)fi);
        stale = want != v.i;
    } else {
        stale = (v.i > 0 && !(v.xi < loga)) || (v.i < v.n - 2 && v.xj < loga);
    }
    if (tm.lane < 4 && stale) {
        const DiscoebSpline& s = table_slot_spline(P, tm.lane);
        if (!v.uniform) {
            want = v.i;
            while (want > 0 && !(DLDG(s.x + want) < loga)) --want;
            while (want < v.n - 2 && DLDG(s.x + want + 1) < loga) ++want;
        }
        load_interval(s, want, v);
    }
    tm.sync();
    const double d = loga - v.xi, B = d * v.rh, A = 1.0 - B;
    const double cubic = __fma_rn(__fma_rn(__dmul_rn(A, A), A, -A), v.Si, __dmul_rn(__fma_rn(__dmul_rn(B, B), B, -B), v.Sj));
    double y = __fma_rn(cubic, v.h26, __fma_rn(A, v.yi, __dmul_rn(B, v.yj)));
    const double slope = __fma_rn(__dmul_rn(v.d2, d), d, __fma_rn(v.d1, d, v.d0));
    if (tm.lane == 4) y = -3.0 * (1.0 + par.w0 + par.wa) * loga + 3.0 * (a - 1.0) * par.wa;
    const double ey = xexp(y);
    if (tm.lane >= 2) y = ey;
    BgTables<double> r;
    r.xe = tm.bcast(y, 0);
    r.xep = tm.bcast(slope, 0);
    r.cs2a = tm.bcast(y, 1);
    r.rhonu = tm.bcast(y, 2);
    r.pnu = tm.bcast(y, 3);
    r.rho_Q = tm.bcast(y, 4);
    return r;
}

// prepare pt for the point (a, t, regime); both helper warps, which meet at barrier 2
__device__ __forceinline__ void prep_point(const WarpTeam& tm, bool warp_a, const DiscoebCosmo& P, const Dims& D,
                                           double k, double a, double t, int regime, Point& pt, int& hint)
{
    if (warp_a) {
        Bg<Dual> bd;
        const Par<Dual> par = make_par<Dual>(P, nullptr);
        const Dual ad(a, 1.0);
        const BgTables<Dual> tb = bg_tables(tm, P, par, (const DiscoebTangent*)nullptr, ad, hint);
        bg_finish(P, par, ad, tb, t, k, regime, bd, Rounding());
        bd.ca2_Q.v = Rounding::ca2(par.wa.v, bd.aH.v, a, bd.w_Q.v, rcp((1.0 + bd.w_Q.v) + 1e-6));
        if (tm.leader()) {
            pt.bd = bd;
            pt.b = bg_value(bd);
            pt.t = t;
            pt.it2 = rcp(t * t);
        }
        tm.sync();
    }
    bar_sync(2, 64);
    if (!warp_a)
        point_functionals(tm, P, D, k, pt);
    else if (tm.leader())
        point_rows(P, k, pt.t, pt);
    tm.sync();
}

// one step attempt of the helper warps: the scale factor through the eight stages, every stage's
// background, then the next point
__device__ __forceinline__ void helper_step(const WarpTeam& tm, bool warp_a, const DiscoebCosmo& P, const Dims& D,
                                            double k, const double* sw, const DiscoebControl& C, Shared& S, int cur,
                                            const ModeMem& M, int bg_count, int& hint, Interval& iv)
{
    // all that is read of the controller's fields, before the first barrier of the attempt
    const double t = S.c.t, h = S.c.h, tnext = S.c.tnext;
    const int regime = S.c.regime, n = D.n, regime_next = regime_at(P, tnext, sw);
    if (warp_a) {
        const Point& pt = S.pt[cur];
        const double igh = rcp(kR5.gamma * h), ih = rcp(h);
        const Dual fa = pt.bd.aH * pt.bd.a;
        const double w00 = igh - fa.d;
        const double y0 = pt.bd.a.v;
        double u0 = y0;
        const double x00 = div_call(fa.v, w00);
        if (tm.leader()) {
            S.st[0].x0 = x00;
            M.K[0] = x00;
            M.sc[SC_W00] = w00;
        }
        // the stage sums' coefficients
        for (int e = tm.lane; e < 64; e += 32) {
            const int s = e >> 3, j = e & 7;
            if (j < s) S.c.cih[s][j] = kR5.C[s][j] * ih;
            if (j == 7 && s < 5) S.c.hd[s] = h * kR5.d[s];
        }
        tm.sync();
        bar_arrive(10, bg_count);
        const Par<double> par = make_par<double>(P, nullptr);
#pragma unroll 1
        for (int s = 1; s < 8; ++s) {
            if (s <= 5) {
                u0 = y0;
                for (int j = 0; j < s; ++j) u0 += kR5.a[s][j] * S.st[j].x0;
            } else {
                u0 = u0 + S.st[s - 1].x0;
            }
            const double ts = __dadd_rn(t, s <= 5 ? __dmul_rn(kR5.c[s], h) : h);  // not fused
            const BgTables<double> tb = stage_tables(tm, P, par, u0, iv);
            Bg<double> b;
            bg_finish(P, par, u0, tb, ts, k, regime, b, Rounding());  // only a'/a is used here
            double r = __dmul_rn(b.aH, b.a);  // f_0, rounded before the sum as where it is stored
            for (int j = 0; j < s; ++j) r += S.c.cih[s][j] * S.st[j].x0;
            const double x0 = div_call(r, w00);
            if (tm.leader()) {
                S.st[s].tb = tb;
                S.st[s].a = u0;
                S.st[s].ts = ts;
                S.st[s].x0 = x0;
                M.K[s * n] = x0;
                if (s == 7) M.u[0] = u0;
            }
            tm.sync();
            bar_sync(2, 64);
        }
        const double an = u0 + S.st[7].x0;
        prep_point(tm, true, P, D, k, an, tnext, regime_next, S.pt[cur ^ 1], hint);
    } else {
        // the controller's powers of the previous errors, known before the attempt ends
        if (tm.lane < 2) {
            const double eo = 6.0, c = tm.lane ? C.dcoeff / eo : -(C.pcoeff + 2.0 * C.dcoeff) / eo;
            S.c.pw[tm.lane] = c == 0.0 ? 1.0 : pow_call(tm.lane ? S.c.e3 : S.c.e2, c);
        }
        const Par<double> par = make_par<double>(P, nullptr);
        for (int s = 1; s < 8; ++s) {
            bar_sync(2, 64);
            Stage& g = S.st[s];
            Bg<double> b;
            bg_finish(P, par, g.a, g.tb, g.ts, k, regime, b, Rounding());
            if (tm.leader()) g.b = b;
            if (tm.lane < D.nq) {
                const double iv = inv_vq(P, b, tm.lane);
                g.iv[tm.lane] = iv;
                g.v[tm.lane] = rcp(iv);
            }
            tm.sync();
            bar_arrive(2 + s, bg_count);
        }
        prep_point(tm, false, P, D, k, 0.0, 0.0, 0, S.pt[cur ^ 1], hint);
    }
}

// ---- the chains ----
// W's rows are kept where the substitutions want them: element p of long chain c (photons from row 8
// on, polarisation, massless neutrinos, momentum bins) at position p nl + c, so that a lane per chain
// walks with one stride and the lanes' accesses are consecutive.  All chains end at p = steps - 1; the
// positions before a shorter chain's first element hold zeros (main diagonal one), whose results are
// zero, so that no lane branches.  Rows 1..7 and the dark-energy pair follow.  The photon-baryon
// chain's rows 5..7, with W's two entries outside the tridiagonal form, (6, 8) and (8, 6), are
// eliminated by its lane around the common loop; that fills nothing else.
struct Bands {
    double* E;  // per position: lower, main (after the factorisation: its reciprocal), upper diagonal,
                // and the right-hand side / solution of a stage
    double* Z;  // A^{-1} U (three columns) and stage 0's right-hand side, pc apart
    int nl, steps, pc, row8;  // chains, positions per chain, positions, row 8's position
};
__device__ __forceinline__ Bands make_bands(const Dims& D, double* mem)
{
    Bands B;
    B.nl = chain_stride(D);
    B.steps = chain_steps(D);
    B.pc = B.steps * B.nl + 9;
    B.row8 = (B.steps - D.lmaxg) * B.nl;
    B.E = mem;
    B.Z = mem + 4 * B.pc;
    return B;
}
enum { E_LO = 0, E_DI = 1, E_UP = 2, E_V = 3 };
__device__ __forceinline__ int position(const Dims& D, const Bands& B, int i)
{
    const int extra = B.steps * B.nl;
    if (i < 8) return extra + i - 1;
    if (i >= D.n - 2) return extra + 7 + i - (D.n - 2);
    if (i < D.idxgp) return (B.steps - D.lmaxg + i - 8) * B.nl;
    if (i < D.idxr) return (B.steps - (D.lmaxgp + 1) + i - D.idxgp) * B.nl + 1;
    if (i < D.iq0) return (B.steps - (D.lmaxr + 1) + i - D.idxr) * B.nl + 2;
    const int l = div_nq(i - D.iq0, D.nq);
    return (B.steps - (D.lmaxnu + 1) + l) * B.nl + 3 + (i - D.iq0 - l * D.nq);
}
// length of long chain c
__device__ __forceinline__ int chain_length(const Dims& D, int c)
{
    return c == 0 ? D.lmaxg : (c == 1 ? D.lmaxgp + 1 : (c == 2 ? D.lmaxr + 1 : D.lmaxnu + 1));
}

// LU of long chain c without pivoting (factor_chain), main diagonal replaced by its reciprocal
__device__ __forceinline__ bool factor_tri(const Bands& B, int c, int len, Ctl& C)
{
    const int extra = B.steps * B.nl;
    bool ok = true;
    auto invert = [&](double piv) {
        ok = ok && fabs(piv) > 0.0 && xfinite(piv);
        return __drcp_rn(piv);
    };
    const int skip = B.steps - len;
    double* e = B.E + 4 * (skip * B.nl + c);
    if (c == 0) {
        double *e5 = B.E + 4 * (extra + 4), *e6 = e5 + 4, *e7 = e5 + 8;
        const double r5 = invert(e5[E_DI]), l6 = e6[E_LO] * r5;
        const double r6 = invert(e6[E_DI] - l6 * e5[E_UP]), l2 = C.al2 * r6, l7 = e7[E_LO] * r6;
        const double r7 = invert(e7[E_DI] - l7 * e6[E_UP]), l8 = e[E_LO] * r7;
        double d8 = e[E_DI] - l2 * C.au2;
        d8 -= l8 * e7[E_UP];
        e5[E_DI] = r5;
        e6[E_LO] = l6;
        e6[E_DI] = r6;
        e7[E_LO] = l7;
        e7[E_DI] = r7;
        e[E_LO] = l8;
        e[E_DI] = d8;
        C.al2 = l2;
    }
    double rp = invert(e[E_DI]), up = e[E_UP];
    e[E_DI] = rp;
    double a = 0.0, d = 0.0, u = 0.0;
    const int st = 4 * B.nl;
    if (len > 1) { a = e[st + E_LO]; d = e[st + E_DI]; u = e[st + E_UP]; }
    for (int p = 1; p < len; ++p) {
        e += st;
        const double l = a * rp, piv = d - l * up;
        up = u;
        if (p + 1 < len) { a = e[st + E_LO]; d = e[st + E_DI]; u = e[st + E_UP]; }
        rp = invert(piv);
        e[E_LO] = l;
        e[E_DI] = rp;
    }
    return ok;
}

// Forward and back substitution along long chain c (solve_chain) for z (elements ZS apart; the factors
// ES apart), with the
// chains' stride NL known at compile time; each element is loaded four steps before its use.
template <int ZS, int NL, int ES>
__device__ __forceinline__ void solve_tri_n(const Bands& B, int c, double al2, double au2, double* z)
{
    constexpr int se = ES * NL, sz = ZS * NL;
    extern __shared__ double smem[];  // (indices into it, so that every access is a shared-memory one)
    int e = (int)(B.E - smem) + ES * c, zp = (int)(z - smem) + ZS * c;
    const int extra = B.steps * NL;
    const double* e5 = B.E + ES * (extra + 4);
    double* z5 = z + ZS * (extra + 4);
    double* z8 = z + ZS * B.row8;
    double v5 = 0.0, v6 = 0.0, v7 = 0.0;
    if (c == 0) {
        v5 = z5[0];
        v6 = z5[ZS] - e5[ES + E_LO] * v5;
        v7 = z5[2 * ZS] - e5[2 * ES + E_LO] * v6;
        double v8 = *z8 - B.E[ES * B.row8 + E_LO] * v7;
        v8 -= al2 * v6;
        *z8 = v8;
    }
    double zz[4], aa[4], dd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        zz[q] = smem[zp + q * sz];
        aa[q] = smem[e + q * se + E_LO];
    }
    double x = 0.0;
#pragma unroll 1
    for (int p = 0; p < B.steps; p += 4) {  // (the last round's loads run into what follows: unused)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x = zz[q] - aa[q] * x;
            smem[zp + q * sz] = x;
            zz[q] = smem[zp + (4 + q) * sz];
            aa[q] = smem[e + (4 + q) * se + E_LO];
        }
        zp += 4 * sz;
        e += 4 * se;
    }
    zp -= 4 * sz;
    e -= 4 * se;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        zz[q] = smem[zp + q * sz];
        aa[q] = smem[e + q * se + E_UP];
        dd[q] = smem[e + q * se + E_DI];
    }
    x = 0.0;
#pragma unroll 1
    for (int p = 0; p < B.steps; p += 4) {  // (and here into what precedes)
#pragma unroll
        for (int q = 3; q >= 0; --q) {
            x = (zz[q] - aa[q] * x) * dd[q];
            smem[zp + q * sz] = x;
            zz[q] = smem[zp + (q - 4) * sz];
            aa[q] = smem[e + (q - 4) * se + E_UP];
            dd[q] = smem[e + (q - 4) * se + E_DI];
        }
        zp -= 4 * sz;
        e -= 4 * se;
    }
    if (c == 0) {
        const double x8 = *z8, x7 = (v7 - e5[2 * ES + E_UP] * x8) * e5[2 * ES + E_DI];
        double x6 = v6 - e5[ES + E_UP] * x7;
        x6 -= au2 * x8;
        x6 *= e5[ES + E_DI];
        z5[2 * ZS] = x7;
        z5[ZS] = x6;
        z5[0] = (v5 - e5[E_UP] * x6) * e5[E_DI];
    }
}
// The same with the number of positions known too: the forward results stay in registers, and every
// load is issued ahead of the dependent arithmetic (20 positions: 1490 -> ~800 cycles).
template <int ZS, int NL, int STEPS, int ES>
__device__ __forceinline__ void solve_tri_s(const Bands& B, int c, double al2, double au2, double* z)
{
    extern __shared__ double smem[];
    constexpr int se = ES * NL, sz = ZS * NL, extra = STEPS * NL;
    const int e = (int)(B.E - smem) + ES * c, zp = (int)(z - smem) + ZS * c;
    const double* e5 = B.E + ES * (extra + 4);
    double* z5 = z + ZS * (extra + 4);
    double* z8 = z + ZS * B.row8;
    double v6 = 0.0, v7 = 0.0;
    const bool photon = c == 0;
    if (photon) {
        const double v5 = z5[0];
        v6 = z5[ZS] - e5[ES + E_LO] * v5;
        v7 = z5[2 * ZS] - e5[2 * ES + E_LO] * v6;
        double v8 = *z8 - B.E[ES * B.row8 + E_LO] * v7;
        v8 -= al2 * v6;
        *z8 = v8;
    }
    double v[STEPS];
    double x = 0.0;
#pragma unroll
    for (int p = 0; p < STEPS; ++p) {
        x = smem[zp + p * sz] - smem[e + p * se + E_LO] * x;
        v[p] = x;
    }
    x = 0.0;
#pragma unroll
    for (int p = STEPS - 1; p >= 0; --p) {
        x = (v[p] - smem[e + p * se + E_UP] * x) * smem[e + p * se + E_DI];
        v[p] = x;
    }
#pragma unroll
    for (int p = 0; p < STEPS; ++p) smem[zp + p * sz] = v[p];
    if (photon) {
        const double v5 = z5[0], x8 = *z8, x7 = (v7 - e5[2 * ES + E_UP] * x8) * e5[2 * ES + E_DI];
        double x6 = v6 - e5[ES + E_UP] * x7;
        x6 -= au2 * x8;
        x6 *= e5[ES + E_DI];
        z5[2 * ZS] = x7;
        z5[ZS] = x6;
        z5[0] = (v5 - e5[E_UP] * x6) * e5[E_DI];
    }
}
template <int ZS, int ES = 4> __device__ __forceinline__ void solve_tri(const Bands& B, int c, double al2, double au2, double* z)
{
    if (B.nl != kNarrow) solve_tri_n<ZS, kWide, ES>(B, c, al2, au2, z);
    else if (B.steps == kLong) solve_tri_s<ZS, kNarrow, kLong, ES>(B, c, al2, au2, z);
    else if (B.steps == kShort) solve_tri_s<ZS, kNarrow, kShort, ES>(B, c, al2, au2, z);
    else solve_tri_n<ZS, kNarrow, ES>(B, c, al2, au2, z);
}

// ---- the special rows and metric functionals (special_part, the momentum bins in a loop) ----
// the state in shared memory as special_block reads it
struct StateAt {
    const double* base;
    __device__ __forceinline__ double operator()(int j) const { return base[j]; }
};
// Sums over the momentum bins of w y_q / v, w y_q v and w y_(nq + q): a lane per sum (and per
// derivative part), each adding its bins in order; coef: 1/v and v of bin q at coef[q], coef[16 + q]
__device__ __forceinline__ double neutrino_sum(const DiscoebCosmo& P, int nq, const double* y, bool flux,
                                               const double* coef, int stride)
{
    double acc = 0.0;
#pragma unroll 1
    for (int q0 = 0; q0 < nq; q0 += 5) {
        double x[5], c[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const int q = q0 + j < nq ? q0 + j : 0;
            const double w = P.wq[q];
            x[j] = flux ? w : w * y[q];
            c[j] = flux ? y[nq + q] : coef[q * stride];
        }
#pragma unroll
        for (int j = 0; j < 5; ++j)
            if (q0 + j < nq) acc = __fma_rn(x[j], c[j], acc);
    }
    return acc;
}
__device__ __forceinline__ void neutrino_sums(const WarpTeam& tm, const DiscoebCosmo& P, int nq, const double* y,
                                              const double* bins, double& drho, double& dp, double& fnu)
{
    const double s = neutrino_sum(P, nq, y, tm.lane == 2, bins + (tm.lane == 1 ? DISCOEB_MAX_NQ : 0), 1);
    drho = tm.bcast(s, 0);
    dp = tm.bcast(s, 1);
    fnu = tm.bcast(s, 2);
}
__device__ __forceinline__ void neutrino_sums(const WarpTeam& tm, const DiscoebCosmo& P, int nq, const double* y,
                                              const Dual* bins, Dual& drho, Dual& dp, Dual& fnu)
{
    // lanes 0, 1: 1/v and its derivative; 2, 3: v; 4: the flux
    const double* c = reinterpret_cast<const double*>(bins + ((tm.lane & 2) ? DISCOEB_MAX_NQ : 0)) + (tm.lane & 1);
    const double s = neutrino_sum(P, nq, y, tm.lane == 4, c, 2);
    drho = Dual(tm.bcast(s, 0), tm.bcast(s, 1));
    dp = Dual(tm.bcast(s, 2), tm.bcast(s, 3));
    fnu = Dual(tm.bcast(s, 4), 0.0);
}

// special_part from the sums over the momentum bins
template <class T, class S, class PR>
__device__ __forceinline__ void special_core(const DiscoebCosmo& P, const Dims& D, const Bg<T>& b, double k, double tau,
                                             StateAt Y, const T& drho, T dp, const T& fnu, T sp[15], T& g0, T& g1,
                                             T& g2)
{
    const int n = D.n, idxr = D.idxr;
    const double k2 = k * k;
    const T Omegac = b.par.Omegam - b.par.Omegab;
    dp = dp * (1.0 / 3.0);
    const S eta = Y(2), deltac = Y(3), thetac = Y(4), deltab = Y(5), thetab = Y(6);
    const S deltag = Y(7), thetag = Y(8), y9 = Y(9);
    const S deltar = Y(idxr), thetar = Y(idxr + 1), yr2 = Y(idxr + 2);
    const S deltaq = Y(n - 2), thetaq = Y(n - 1);
    const T rQa2 = PR::product(b.rho_Q, b.a2);
    const T dgm = b.par.grhom * (Omegac * deltac + b.par.Omegab * deltab) * b.ia;
    const T dgnu = P.grhor * P.Nmnu * drho * b.ia2;
    const T dgq = b.par.grhom * b.par.OmegaDE * deltaq * rQa2;
    const T dgrho = dgm + (P.grhog * deltag + P.grhor * P.Neff * deltar) * b.ia2 + dgnu + dgq;
    const T dgrho_wo_rel = dgm + dgnu + dgq;
    T H, thg, thr, dge, dre;
    if (b.rsa) {
        const double sk2 = k2 > 1e-30 ? k2 : 1e-30;
        H = (2.0 * k2 * eta + dgrho_wo_rel) * b.iaHG;
        dre = (4.0 / sk2) * (b.aH * H - sk2 * eta);
        dge = dre + (4.0 / 3.0) * b.rsa_fac * (thetab + 0.5 * H);
        thg = PR::rsa_theta(H, b.rsa_fac, -b.rsa_tcs * (thetab + 0.5 * H) + PR::rsa_inner(-b.aH, thetab, b.cs2 * sk2, deltab, sk2, eta));
        thr = -0.5 * H;
    } else {
        H = (2.0 * k2 * eta + dgrho) * b.iaHG;
        dge = deltag;
        dre = deltar;
        thg = thetag;
        thr = thetar;
    }
    const T rptq = b.opw * b.par.grhom * b.par.OmegaDE * thetaq * rQa2;
    const T dgtheta = b.par.grhom * (Omegac * thetac + b.par.Omegab * thetab) * b.ia +
                (4.0 / 3.0) * (P.grhog * thg + P.Neff * P.grhor * thr) * b.ia2 + P.Nmnu * P.grhor * k * fnu * b.ia2 +
                rptq;
    const T E = (0.5 / k2) * dgtheta;
    const double cs2Q = P.cs2_DE;
    const T dgpres = (P.grhog * dge + P.grhor * P.Neff * dre) * b.ia2 * (1.0 / 3.0) + P.grhor * P.Nmnu * dp * b.ia2 +
                     (cs2Q * b.par.grhom * b.par.OmegaDE * deltaq * rQa2 + (cs2Q - b.ca2_Q) * (3.0 * b.aH * rptq * (1.0 / k2)));
    const bool hier_photons = !b.rsa && !b.tca;
    const T polter = hier_photons ? T(y9 + Y(D.idxgp) + Y(D.idxgp + 2)) : T(0.0);
    const T alpha = (H + 6.0 * E) * (0.5 / k2);
    // special rows
    sp[0] = b.aH * b.a;
    sp[1] = -(dgrho + 3.0 * dgpres) * b.a;
    sp[2] = E;
    sp[3] = -thetac - 0.5 * H;
    sp[4] = -b.aH * thetac;
    sp[5] = -thetab - 0.5 * H;
    sp[6] = -b.aH * thetab + k2 * b.cs2 * deltab + b.po * (thg - thetab);
    if (!b.rsa) {
        sp[7] = (4.0 / 3.0) * (-thg - 0.5 * H);
        sp[8] = k2 * (0.25 * dge - 0.5 * y9) - b.opac * (thg - thetab);
        sp[9] = (8.0 / 15.0) * (thg + k2 * alpha) - 0.6 * k * Y(10) - b.opac * (y9 - 0.1 * polter);
        sp[10] = (4.0 / 3.0) * (-thr - 0.5 * H);
        sp[11] = k2 * (0.25 * dre - 0.5 * yr2);
        sp[12] = b.ufa ? -1.5 * (tau > 1e-30 ? b.itau : 1e30) * yr2 + (4.0 / 15.0) * (thr + 0.5 * H)
                       : (8.0 / 15.0) * (thr + k2 * alpha) - 0.6 * k * Y(idxr + 3);
    } else {
        for (int q = 7; q < 13; ++q) sp[q] = 0.0;
    }
    if (b.de_frozen) {
        sp[13] = 0.0;
        sp[14] = 0.0;
    } else {
        sp[13] = -b.opw * (thetaq + 0.5 * H) - 3.0 * (cs2Q - b.w_Q) * b.aH * deltaq -
                 9.0 * b.opw * (cs2Q - b.ca2_Q) * b.aH * b.aH * (1.0 / k2) * thetaq;
        sp[14] = -(1.0 - 3.0 * cs2Q) * b.aH * thetaq + cs2Q * b.iopw * k2 * deltaq;
    }
    g0 = H;
    g1 = E;
    g2 = polter;
}

template <class T, class S, class PR>
__device__ __forceinline__ void special_block(const WarpTeam& tm, const DiscoebCosmo& P, const Dims& D, const Bg<T>& b,
                                              double k, double tau, StateAt Y, const T* bins, T sp[15], T& g0, T& g1,
                                              T& g2)
{
    T drho = 0.0, dp = 0.0, fnu = 0.0;
    neutrino_sums(tm, P, D.nq, Y.base + D.iq0, bins, drho, dp, fnu);
    special_core<T, S, PR>(P, D, b, k, tau, Y, drho, dp, fnu, sp, g0, g1, g2);
}

// ---- one row per thread: warps "rows" (hierarchy rows) and the lanes of "special" ----

// what never changes of a hierarchy row's coefficients (hier_coef)
struct HierRow {
    int i, im, ip, q;      // row, the rows its lower and upper coefficients read, momentum bin
    bool massive, opaque, trunc, rsa0, ufa0, live;
    double al, au, L1, u0, u1, c2;
};
__device__ __forceinline__ HierRow make_hier_row(const Dims& D, int hh, const double* dlq)
{
    HierRow R;
    R.live = hh < n_hier_rows(D);
    const int i = hier_row(D, R.live ? hh : 0);
    int l, L, species;
    if (i <= 7 + D.lmaxg) { l = i - 7; L = D.lmaxg; species = 0; }
    else if (i <= D.idxgp + D.lmaxgp) { l = i - D.idxgp; L = D.lmaxgp; species = 1; }
    else if (i <= D.idxr + D.lmaxr) { l = i - D.idxr; L = D.lmaxr; species = 2; }
    else { l = div_nq(i - D.iq0, D.nq); L = D.lmaxnu; species = 3; }
    R.massive = species == 3;
    const int st = R.massive ? D.nq : 1;
    R.trunc = l == L;
    R.i = i;
    R.im = i - st;
    R.ip = R.trunc ? i : i + st;
    R.q = hier_bin(D, i);
    R.opaque = species <= 1;
    R.rsa0 = species <= 2;
    R.ufa0 = species == 2;
    const double io = inv_odd(l), dl = dlq[R.q];
    R.al = (double)l * io;
    R.au = (l + 1.0) * io;
    R.L1 = L + 1.0;
    R.c2 = species == 1 ? (l == 0 ? 0.5 : (l == 2 ? 0.1 : 0.0)) : 0.0;
    R.u0 = R.massive ? (l == 0 ? dl * (1.0 / 6.0) : (l == 2 ? -dl * (1.0 / 15.0) : 0.0)) : 0.0;
    R.u1 = (R.massive && l == 2) ? -0.4 * dl : 0.0;
    return R;
}
__device__ __forceinline__ void hier_now(const HierRow& R, const Bg<double>& b, double k, double vq, double& lo,
                                         double& di, double& up, double& u2)
{
    const double scale = R.massive ? k * vq : k;
    lo = R.trunc ? scale : scale * R.al;
    up = R.trunc ? 0.0 : -scale * R.au;
    di = __dadd_rn(R.opaque ? -b.opac : 0.0, R.trunc ? -__dmul_rn(R.L1, b.itau) : -0.0);
    u2 = R.c2 * b.opac;
    if ((R.rsa0 && b.rsa) || (R.ufa0 && b.ufa)) {
        lo = 0.0;
        di = 0.0;
        up = 0.0;
        u2 = 0.0;
    }
}

__device__ __forceinline__ double hier_sum(double lo, double di, double up, double ym, double y, double yp)
{
    return __fma_rn(up, yp, __fma_rn(lo, ym, __dmul_rn(di, y)));
}
// the same row in dual numbers at a plain state (direction: the scale factor)
__device__ __forceinline__ Dual hier_dual(const HierRow& R, const Bg<Dual>& b, double k, const Dual& vq, double ym,
                                          double y, double yp, const double* g, const double* gd)
{
    const bool frozen = (R.rsa0 && b.rsa) || (R.ufa0 && b.ufa);
    const double sv = R.massive ? __dmul_rn(k, vq.v) : k, sd = R.massive ? __dmul_rn(k, vq.d) : 0.0;
    double lov = R.trunc ? sv : __dmul_rn(sv, R.al), lod = R.trunc ? sd : __dmul_rn(sd, R.al);
    double upv = R.trunc ? 0.0 : __dmul_rn(-sv, R.au), upd = R.trunc ? 0.0 : __dmul_rn(-sd, R.au);
    double div = __dadd_rn(R.opaque ? -b.opac.v : 0.0, R.trunc ? -__dmul_rn(R.L1, b.itau) : -0.0);
    double did = R.opaque ? -b.opac.d : 0.0;
    double u2v = __dmul_rn(R.c2, b.opac.v), u2d = __dmul_rn(R.c2, b.opac.d);
    if (frozen) lov = lod = upv = upd = div = did = u2v = u2d = 0.0;
    double v = hier_sum(lov, div, upv, ym, y, yp), d = hier_sum(lod, did, upd, ym, y, yp);
    v = __fma_rn(u2v, g[2], __fma_rn(R.u1, g[1], __fma_rn(R.u0, g[0], v)));
    d = __dadd_rn(__dadd_rn(d, __dmul_rn(R.u0, gd[0])), __dmul_rn(R.u1, gd[1]));
    d = __dadd_rn(d, __fma_rn(u2d, g[2], __dmul_rn(u2v, gd[2])));
    return Dual(v, d);
}

// r = f + h d_s dT + sum C_sj K_j / h, with the scale factor's column removed
template <int s>
__device__ __forceinline__ double stage_rhs_at(const Ctl& C, const double* Ki, int n, double f, double dT, double col0,
                                               double x0)
{
    double kk[7], c[7];
#pragma unroll
    for (int j = 0; j < s; ++j) {
        kk[j] = Ki[j * n];
        c[j] = C.cih[s][j];
    }
    double r = f;
    if (s < 5) r += C.hd[s] * dT;
#pragma unroll
    for (int j = 0; j < s; ++j) r += c[j] * kk[j];
    r += col0 * x0;
    return r;
}
__device__ __forceinline__ double stage_rhs(const Ctl& C, const double* Ki, int n, int s, double f, double dT,
                                            double col0, double x0)
{
    switch (s) {
    case 0: return stage_rhs_at<0>(C, Ki, n, f, dT, col0, x0);
    case 1: return stage_rhs_at<1>(C, Ki, n, f, dT, col0, x0);
    case 2: return stage_rhs_at<2>(C, Ki, n, f, dT, col0, x0);
    case 3: return stage_rhs_at<3>(C, Ki, n, f, dT, col0, x0);
    case 4: return stage_rhs_at<4>(C, Ki, n, f, dT, col0, x0);
    case 5: return stage_rhs_at<5>(C, Ki, n, f, dT, col0, x0);
    case 6: return stage_rhs_at<6>(C, Ki, n, f, dT, col0, x0);
    default: return stage_rhs_at<7>(C, Ki, n, f, dT, col0, x0);
    }
}
template <int s> __device__ __forceinline__ double stage_state_at(const double* Ki, int n, double y)
{
    double kk[5];
#pragma unroll
    for (int j = 0; j < s; ++j) kk[j] = Ki[j * n];
    double v = y;
#pragma unroll
    for (int j = 0; j < s; ++j) v += kR5.a[s][j] * kk[j];
    return v;
}
__device__ __forceinline__ double stage_state(const double* Ki, int n, int s, double y, double u)
{
    switch (s) {
    case 1: return stage_state_at<1>(Ki, n, y);
    case 2: return stage_state_at<2>(Ki, n, y);
    case 3: return stage_state_at<3>(Ki, n, y);
    case 4: return stage_state_at<4>(Ki, n, y);
    case 5: return stage_state_at<5>(Ki, n, y);
    default: return u + Ki[(s - 1) * n];
    }
}

// the positions of the state slots a lane adds up for the functionals G and F1, and its G and F1
struct Slots {
    int j0, j1, ns;
};
__device__ __forceinline__ Slots make_slots(const Dims& D, const Bands& B, int lane)
{
    const int ns = n_slots(D);
    return Slots{lane < ns ? position(D, B, slot_index(D, lane)) : 0,
                 lane + 32 < ns ? position(D, B, slot_index(D, lane + 32)) : 0, ns};
}
struct SlotG {
    double g[4], h[4];
};
__device__ __forceinline__ SlotG load_slots(const Slots& sl, int lane, const ModeMem& M)
{
    SlotG G;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const double* g = M.Gs + r * kMaxSlots;  // F1s follows the three rows of Gs
        G.g[r] = lane < sl.ns ? g[lane] : 0.0;
        G.h[r] = lane + 32 < sl.ns ? g[lane + 32] : 0.0;
    }
    return G;
}
// the functionals (h', eta', polter) and F1 of z: sums over the lanes, each the same tree as
// WarpTeam::sum; every lane gets all four.  The lanes share the four trees out: the first two levels
// halve what a lane still adds.
template <int ZS>
__device__ __forceinline__ void slot_sums(const WarpTeam& tm, const Slots& sl, const SlotG& G, const double* z,
                                          double out[4])
{
    const double v = tm.lane < sl.ns ? z[ZS * sl.j0] : 0.0;
    double a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = G.g[r] * v;
    if (sl.ns > 32) {
        const double w = tm.lane + 32 < sl.ns ? z[ZS * sl.j1] : 0.0;
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] += G.h[r] * w;
    }
    const bool up = (tm.lane & 16) != 0, up2 = (tm.lane & 8) != 0;
    const double s0 = up ? a[0] : a[2], s1 = up ? a[1] : a[3];
    double b0 = up ? a[2] : a[0], b1 = up ? a[3] : a[1];
    b0 += __shfl_xor_sync(0xffffffffu, s0, 16);
    b1 += __shfl_xor_sync(0xffffffffu, s1, 16);
    const double s2 = up2 ? b0 : b1;
    double c = up2 ? b1 : b0;
    c += __shfl_xor_sync(0xffffffffu, s2, 8);
    c += __shfl_xor_sync(0xffffffffu, c, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
#pragma unroll
    for (int r = 0; r < 4; ++r) out[r] = __shfl_sync(0xffffffffu, c, 8 * r);
}

// the two short chains: CDM (rows 3, 4) and dark energy
template <int ES = 4> __device__ __forceinline__ double* short_chain(const Bands& B, int which)
{
    return B.E + ES * (B.steps * B.nl + (which ? 7 : 2));
}
template <int ZS, int ES = 4> __device__ __forceinline__ void solve_short(const Bands& B, int lane, double* z, int nrhs)
{
    if (lane < 2 * nrhs) {
        const double* c = short_chain<ES>(B, lane & 1);
        double* v = z + (lane >> 1) * B.pc + ZS * (B.steps * B.nl + ((lane & 1) ? 7 : 2));
        const double b = v[ZS] - c[ES + E_LO] * v[0];
        const double x1 = b * c[ES + E_DI];
        v[ZS] = x1;
        v[0] = (v[0] - c[E_UP] * x1) * c[E_DI];
    }
}

// what a row thread carries through the solve; i < 0: none
struct RowState {
    int i, pos;
    double y, dT, col0, f, u;
};

// One step attempt of special + rows.  Returns false (in every thread) on a singular factorisation.
__device__ __forceinline__ bool row_step(const WarpTeam& tm, bool special, int wr, int n_row_warps, const HierRow& H,
                                         const Slots& sl, const DiscoebCosmo& P, const Dims& D, double k, Shared& S,
                                         const Point& pt, const ModeMem& M, const Bands& B, RowState& R)
{
    const int n = D.n, nq = D.nq;
    const int c_rows = 32 * (1 + n_row_warps), c_bg = c_rows + 32, c_all = c_rows + 32;
    const double t = S.c.t, h = S.c.h;
    const bool fresh = S.c.fresh != 0;
    const double gh = kR5.gamma * h;
    const double igh = rcp(gh);
    const int i = R.i;
    double* Ki = M.K + (i < 0 ? 0 : i);
    double* e = B.E + 4 * R.pos;
    double* zc = B.Z + R.pos;
    // W's rows and U; the explicit tau derivative; the dual right-hand side of the special rows
    if (special) {
        if (i >= 1) {
            const int m = tm.lane;
            e[E_LO] = -pt.row[m][0];
            e[E_DI] = -pt.row[m][1] + igh;
            e[E_UP] = -pt.row[m][2];
            if (i == 6) S.c.au2 = -pt.s68;
            if (i == 8) S.c.al2 = -pt.s86;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                double z = pt.row[m][3 + r];
                if (i == 2) z *= gh;
                if (i == 6) z += pt.etac * (pt.row[2][3 + r] * gh);
                zc[r * B.pc] = z;
            }
            // (row r's explicit tau term: the fluid closure's)
            if (fresh) R.dT = (m == 12 && pt.b.ufa && t > 1e-30) ? 1.5 * pt.it2 * M.y[i] : 0.0;
        }
        if (fresh) {
            for (int q = tm.lane; q < sl.ns; q += 32) {
                M.Gs[q] = pt.Gs[q];
                M.Gs[kMaxSlots + q] = pt.Gs[kMaxSlots + q];
                M.Gs[2 * kMaxSlots + q] = pt.Gs[2 * kMaxSlots + q];
                M.F1s[q] = pt.F1s[q];
            }
        }
    } else if (H.live) {
        double lo, di, up, u2;
        hier_now(H, pt.b, k, pt.vf[H.q], lo, di, up, u2);
        e[E_LO] = -lo;
        e[E_DI] = igh - di;
        e[E_UP] = -up;
        zc[0] = H.u0;
        zc[B.pc] = H.u1;
        zc[2 * B.pc] = u2;
        // the truncation rows' explicit tau term
        if (fresh)
            R.dT = (H.trunc && !((H.rsa0 && pt.b.rsa) || (H.ufa0 && pt.b.ufa))) ? H.L1 * pt.it2 * M.y[i] : 0.0;
    }
    bar_sync(11, c_all);
    // (chains: factorisation)  the dual right-hand side, stage 0's r
    bool ok = true;
    if (special) {
        if (tm.lane < 2) {
            double* c = short_chain(B, tm.lane);
            const double p0 = c[E_DI], r0 = rcp(p0), l1 = c[4 + E_LO] * r0, p1 = c[4 + E_DI] - l1 * c[E_UP];
            ok = fabs(p0) > 0.0 && xfinite(p0) && fabs(p1) > 0.0 && xfinite(p1);
            c[E_DI] = r0;
            c[4 + E_LO] = l1;
            c[4 + E_DI] = rcp(p1);
        }
        if (fresh) {
            Dual sp[15], g0, g1, g2;
            const StateAt Y{M.y};
            Bg<Dual> bd = pt.bd;  // with the derivatives known at compile time
            bd.par = make_par<Dual>(P, nullptr);
            bd.a.d = 1.0;
            special_block<Dual, double, Rounding>(tm, P, D, bd, k, t, Y, pt.iv, sp, g0, g1, g2);
            Rounding::shear_rows(D, pt.b, k, t, Y, g0.v, g1.v, g2.v, sp[9].v, sp[12].v);
            if (tm.leader()) {
#pragma unroll
                for (int ss = 0; ss < 15; ++ss) {
                    const int r = special_row(D, ss);
                    M.f[r] = sp[ss].v;
                    M.col0[r] = sp[ss].d;
                }
                S.c.g[0] = g0.v; S.c.g[1] = g1.v; S.c.g[2] = g2.v;
                S.c.gd[0] = g0.d; S.c.gd[1] = g1.d; S.c.gd[2] = g2.d;
            }
            tm.sync();
            if (tm.lane < 15) {
                R.f = M.f[i];
                R.col0 = M.col0[i];
            }
        }
    }
    if (fresh) bar_sync(1, c_rows);
    if (!special && fresh && H.live) {
        const Dual fi = hier_dual(H, pt.bd, k, nq > 0 ? pt.v[H.q] : Dual(1.0), M.y[H.im], M.y[i], M.y[H.ip], S.c.g,
                                  S.c.gd);
        R.f = fi.v;
        R.col0 = fi.d;
        M.f[i] = fi.v;
        M.col0[i] = fi.d;
    }
    if (!ok) S.c.fac_ok = 0;
    bar_sync(10, c_bg);
    // a special lane's stage value into the chains' right-hand side
    auto put_special = [&](double v, double* to) {
        if (i == 2) v *= gh;
        const double v2 = tm.bcast(v, 2);
        if (i == 6) v += pt.etac * v2;
        if (i >= 1) *to = v;
    };
    {
        double v = 0.0;
        if (i >= 1) v = stage_rhs(S.c, Ki, n, 0, R.f, R.dT, R.col0, S.st[0].x0);
        if (special) put_special(v, zc + 3 * B.pc);
        else if (H.live) zc[3 * B.pc] = v;
    }
    bar_sync(11, c_all);
    if (special) solve_short<1>(B, tm.lane, B.Z, 4);
    bar_sync(11, c_all);
    // C = I - G Z and F1 Z (rows), G and F1 of stage 0 (special)
    const SlotG G = load_slots(sl, tm.lane, M);
    if (special) {
        double o[4];
        slot_sums<1>(tm, sl, G, B.Z + 3 * B.pc, o);
        if (tm.leader())
            for (int v = 0; v < 4; ++v) S.c.gz0[v] = o[v];
    } else {
        for (int s = wr; s < 3; s += n_row_warps) {  // column s of G Z and F1 Z
            double o[4];
            slot_sums<1>(tm, sl, G, B.Z + s * B.pc, o);
            if (tm.leader()) {
                for (int r = 0; r < 3; ++r) S.c.cmat[3 * r + s] = (r == s ? 1.0 : 0.0) - o[r];
                M.sc[SC_F1Z + s] = o[3];
            }
        }
    }
    bar_sync(1, c_rows);
    const double* C = S.c.cmat;
    // 3x3 inverse by cofactors
    auto minor = [](double a, double d, double b, double c) {
        return __fma_rn(a, d, -__dmul_rn(b, c));
    };
    const double c00 = minor(C[4], C[8], C[5], C[7]);
    const double c01 = minor(C[5], C[6], C[3], C[8]);
    const double c02 = minor(C[3], C[7], C[4], C[6]);
    const double det = __fma_rn(C[2], c02, __fma_rn(C[0], c00, __dmul_rn(C[1], c01)));
    const double id = rcp(det);
    double Ci[9];
    Ci[0] = c00 * id;
    Ci[1] = minor(C[2], C[7], C[1], C[8]) * id;
    Ci[2] = minor(C[1], C[5], C[2], C[4]) * id;
    Ci[3] = c01 * id;
    Ci[4] = minor(C[0], C[8], C[2], C[6]) * id;
    Ci[5] = minor(C[2], C[3], C[0], C[5]) * id;
    Ci[6] = c02 * id;
    Ci[7] = minor(C[1], C[6], C[0], C[7]) * id;
    Ci[8] = minor(C[0], C[4], C[1], C[3]) * id;
    if (special && tm.leader())
        for (int q = 0; q < 9; ++q) M.sc[SC_CINV + q] = Ci[q];
    const bool good = S.c.fac_ok != 0 && xfinite(det) && det != 0.0;
    // K_s of this thread's row from the chains' solution and the rank-3 coupling; row 1 (a h', read by
    // no equation) is the functional F1
    const double z0 = i == 1 ? M.sc[SC_F1Z] + pt.f1u[0] : zc[0], z1 = i == 1 ? M.sc[SC_F1Z + 1] + pt.f1u[1] : zc[B.pc],
                 z2 = i == 1 ? M.sc[SC_F1Z + 2] + pt.f1u[2] : zc[2 * B.pc];
    const double scale = i == 1 ? gh : 1.0;
    auto finish = [&](int s, const double* gz, double v) {
        const double c0 = Ci[0] * gz[0] + Ci[1] * gz[1] + Ci[2] * gz[2];
        const double c1 = Ci[3] * gz[0] + Ci[4] * gz[1] + Ci[5] * gz[2];
        const double c2 = Ci[6] * gz[0] + Ci[7] * gz[1] + Ci[8] * gz[2];
        if (i == 1) v += gz[3];
        if (i >= 1) Ki[s * n] = scale * (v + (z0 * c0 + z1 * c1 + z2 * c2));
    };
    finish(0, S.c.gz0, zc[3 * B.pc]);
#pragma unroll 1
    for (int s = 1; s < 8; ++s) {
        if (i >= 1) {
            R.u = stage_state(Ki, n, s, R.y, R.u);
            M.u[i] = R.u;
        }
        bar_sync(1, c_rows);
        bar_sync(2 + s, c_bg);
        const Stage& g = S.st[s];
        const double x0 = g.x0;
        double f = 0.0, u2 = 0.0;
        if (special) {
            double sp[15], g0, g1, g2;
            const StateAt Y{M.u};
            special_block<double, double, Rounding>(tm, P, D, g.b, k, g.ts, Y, g.iv, sp, g0, g1, g2);
            Rounding::shear_rows(D, g.b, k, g.ts, Y, g0, g1, g2, sp[9], sp[12]);
            if (tm.leader()) {
                S.c.g[0] = g0; S.c.g[1] = g1; S.c.g[2] = g2;
#pragma unroll
                for (int ss = 0; ss < 15; ++ss) S.c.sp[ss] = sp[ss];
            }
            tm.sync();
            if (tm.lane < 15) f = S.c.sp[tm.lane];
        } else if (H.live) {
            double lo, di, up;
            hier_now(H, g.b, k, g.v[H.q], lo, di, up, u2);
            f = hier_sum(lo, di, up, M.u[H.im], M.u[i], M.u[H.ip]);
        }
        bar_sync(1, c_rows);
        if (!special) f = __fma_rn(u2, S.c.g[2], __fma_rn(H.u1, S.c.g[1], __fma_rn(H.u0, S.c.g[0], f)));
        double v = 0.0;
        if (i >= 1) v = stage_rhs(S.c, Ki, n, s, f, R.dT, R.col0, x0);
        if (special) put_special(v, e + E_V);
        else if (H.live) e[E_V] = v;
        bar_sync(11, c_all);
        if (special) solve_short<4>(B, tm.lane, B.E + E_V, 1);
        bar_sync(11, c_all);
        double gz[4];
        slot_sums<4>(tm, sl, G, B.E + E_V, gz);
        finish(s, gz, e[E_V]);
    }
    return good;
}

// one step attempt of the chains warp
__device__ __forceinline__ void chain_step(const WarpTeam& tm, const Dims& D, Shared& S, const Bands& B, int c_all)
{
    bar_sync(11, c_all);
    const int nc = 3 + D.nq;
    if (tm.lane < nc && !factor_tri(B, tm.lane, chain_length(D, tm.lane), S.c)) S.c.fac_ok = 0;
    bar_sync(11, c_all);
    const double al2 = S.c.al2, au2 = S.c.au2;
    for (int x = tm.lane; x < 4 * nc; x += 32) {
        const int r = x / nc;
        solve_tri<1>(B, x - r * nc, al2, au2, B.Z + r * B.pc);
    }
    bar_sync(11, c_all);
#pragma unroll 1
    for (int s = 1; s < 8; ++s) {
        bar_sync(11, c_all);
        if (tm.lane < nc) solve_tri<4>(B, tm.lane, al2, au2, B.E + E_V);
        bar_sync(11, c_all);
    }
}

// publish() of a solve whose steps nobody records
struct NoPublish {
    __device__ __forceinline__ void copy(int, double, const ModeMem&, const Bands&, int, int) const {}
    __device__ __forceinline__ void done(const ModeMem&) const {}
};

// The solve.  y0 is in M.y; emit(j, y) runs on warp 0 with the state exactly at tout[j];
// rows(j, i, y_i) runs on the thread that owns row i (either may do nothing); accept as in
// solve_mode, on warp 0.  After an accepted step, publish.copy(row, y, M, B, thread, threads) runs on
// every thread of special + rows while M still holds the step (all but row 0, whose next stages are
// under way), and publish.done(M) on warp 0 when all of them are through.  Every thread of the block
// calls it; the result is valid on warp 0.
template <class Emit, class Rows, class Accept, class Publish = NoPublish>
__device__ __forceinline__ SolveResult solve_mode_block(const DiscoebCosmo& P, const Dims& D, const DiscoebControl& C,
                                                        double k, double t0, const double* sw, int nout,
                                                        const double* tout, const ModeMem& M, Shared& S, Emit& emit,
                                                        Rows& rows, Accept& accept,
                                                        const Publish& publish = Publish())
{
    const int warp = threadIdx.x >> 5;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int n = D.n, nrw = row_warps(D);
    const int c_rows = 32 * (1 + nrw), c_all = c_rows + 32, c_solve = c_all + 64;
    const Bands B = make_bands(D, M.A);
    SolveResult R = {DISCOEB_OK, 0, 0, 0};
    int hint = P.xe_loga.n_knots / 2;
    int cur = 0;
    if (warp == 2 + nrw && tm.lane < 2) S.pt[tm.lane].regime = -1;
    if (threadIdx.x < DISCOEB_MAX_NQ) S.c.dlq[threadIdx.x] = (int)threadIdx.x < D.nq ? dlfdlq_of(P.q[threadIdx.x]) : 0.0;
    if (warp >= 2 + nrw) {  // scale and prep
        const bool scale = warp == 2 + nrw;
        Interval iv;
        init_interval(tm, P, iv);
        bar_sync(2, 64);
        prep_point(tm, scale, P, D, k, M.y[0], t0, regime_at(P, t0, sw), S.pt[0], hint);
        for (;;) {
            bar_sync(0, c_solve);
            if (!S.c.go) break;
            if (S.c.accepted) cur ^= 1;
            helper_step(tm, scale, P, D, k, sw, C, S, cur, M, c_rows + 32, hint, iv);
        }
        return R;
    }
    if (warp == 1) {  // chains
        for (int x = tm.lane; x < 4 * B.pc; x += 32) {  // (the positions before the chains)
            B.E[x] = (x & 3) == E_DI ? 1.0 : 0.0;
            B.Z[x] = 0.0;
        }
        for (;;) {
            bar_sync(0, c_solve);
            if (!S.c.go) break;
            chain_step(tm, D, S, B, c_all);
        }
        return R;
    }
    bar_sync(1, c_rows);  // S.c.dlq
    const bool special = warp == 0;
    const HierRow H = make_hier_row(D, special ? 0 : 32 * (warp - 2) + tm.lane, S.c.dlq);
    const Slots sl = make_slots(D, B, tm.lane);
    RowState W;
    W.i = special ? (tm.lane < 15 ? special_row(D, tm.lane) : -1) : (H.live ? H.i : -1);
    W.pos = W.i >= 1 ? position(D, B, W.i) : B.steps * B.nl;
    W.y = W.i >= 0 ? M.y[W.i] : 0.0;
    W.dT = W.col0 = W.f = W.u = 0.0;
    double t1 = tout[0];
    for (int j = 1; j < nout; ++j) t1 = tout[j] > t1 ? tout[j] : t1;
    const double eo = 6.0;  // diffrax error order of a 5th-order method: order + 1
    const double c1 = (C.icoeff + C.pcoeff + C.dcoeff) / eo;
    double prev_inv = 1.0, prev_prev_inv = 1.0;
    double t = t0;
    double dt = fmin(t0 / 4.0, 0.5 * (t1 - t0));  // dt0 of perturbations.py:910
    double dt_try = dt;
    int iout = 0;
    double t_out = tout[0];  // tout[iout]
    bool clipped = false, first = true, keep = false, ok = true;
    for (;;) {
        if (warp == 0) {
            // the controller: the previous attempt's outcome, then the next attempt
            int go = 1;
            keep = false;
            if (!first) {
                R.steps++;
                const double h = S.c.h;
                double e = 0.0;
                if (tm.lane < 6) {
                    const int q = tm.lane, i = q == 0 ? 0 : (q < 3 ? q + 1 : q + 2);  // 0, 2, 3, 5, 6, 7
                    const double w = q == 1 ? k * k : (q == 4 ? rcp(k * k) : 1.0);
                    const double y1 = M.u[i] + M.K[7 * n + i];
                    const double sc = fmax(fabs(M.y[i]), fabs(y1));
                    e = div_call(M.K[7 * n + i], C.atol + C.rtol * sc) * w;
                }
                double sumsq = 0.0;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const double eq = tm.bcast(e, q);
                    sumsq += eq * eq;
                }
                const double nbad = (double)S.c.nbad_cand + 1024.0 * (double)S.c.nbad_start;
                if (nbad >= 1024.0) {  // no step size can help
                    R.status = DISCOEB_NONFINITE;
                    go = 0;
                } else {
                    const bool finite = ok && nbad == 0.0;
                    const double err = finite ? xsqrt(div_call(sumsq, 6.0)) : INFINITY;
                    keep = err < 1.0;
                    double inv = rcp(err);
                    const double f1 = pow_call(inv, c1);
                    const double f2 = S.c.pw[0], f3 = S.c.pw[1];
                    const double fmn = keep ? 1.0 : C.factormin;
                    double factor = 0.9 * f1 * f2 * f3;
                    if (!(factor == factor)) factor = fmn;
                    factor = fmin(fmax(factor, fmn), C.factormax);
                    if (inv == 0.0 || !xfinite(inv)) inv = 1.0;
                    double dtn = h * factor;
                    if (keep) {
                        if (!accept(t, h, S.c.tnext, S.c.regime)) {
                            R.status = DISCOEB_ABORTED;
                            go = 0;
                            keep = false;
                        } else {
                            R.accepted++;
                            t = S.c.tnext;
                            if (clipped && dt_try > dtn) dtn = dt_try;
                            prev_prev_inv = prev_inv;
                            prev_inv = inv;
                        }
                    }
                    dt = dtn;
                }
            }
            double h = 0.0, tnext = 0.0;
            int iout_next = iout;
            double tn_out = t_out;
            if (keep)
                while (iout_next < nout && tn_out <= t) {
                    iout_next++;
                    if (iout_next < nout) tn_out = tout[iout_next];
                }
            if (go && !(t < t1)) go = 0;
            if (go && R.steps >= C.max_steps) {
                R.status = DISCOEB_MAX_STEPS;
                go = 0;
            }
            if (go) {
                double tev = t1;
                if (iout_next < nout && tn_out < tev) tev = tn_out;
                for (int q = 0; q < 3; ++q)
                    if (sw[q] > t && sw[q] < tev) tev = sw[q];
                dt_try = dt;
                tnext = t + dt;
                clipped = false;
                if (tnext >= tev - 1e-12 * fabs(tev)) { clipped = tnext > tev; tnext = tev; }
                h = tnext - t;
                if (!(h > 1e-14 * fabs(t))) {
                    R.status = DISCOEB_DT_UNDERFLOW;
                    go = 0;
                }
            }
            tm.sync();  // every lane has read the previous attempt's fields
            if (tm.leader()) {
                if (go) {
                    S.c.t = t;
                    S.c.h = h;
                    S.c.tnext = tnext;
                }
                if (go) S.c.regime = regime_at(P, t, sw);
                S.c.go = go;
                S.c.fresh = first || keep;
                S.c.accepted = keep;
                S.c.nbad_cand = 0;
                S.c.nbad_start = 0;
                S.c.fac_ok = 1;
                S.c.e2 = prev_inv;
                S.c.e3 = prev_prev_inv;
                // the scale warp overwrites its stages while the rows advance
                if (keep) S.c.y0_next = M.u[0] + M.K[7 * n];
            }
        }
        bar_sync(0, c_solve);
        first = false;
        const int go = S.c.go, accepted = S.c.accepted;
        if (accepted) {
            cur ^= 1;
            publish.copy(W.i, W.y, M, B, special ? tm.lane : 32 * (warp - 1) + tm.lane, c_rows);
            // the state advances; each thread its own row
            if (W.i >= 0) {
                W.y = W.i == 0 ? S.c.y0_next : W.u + M.K[7 * n + W.i];
                M.y[W.i] = W.y;
            }
            bar_sync(1, c_rows);
            if (special) publish.done(M);
            const double tacc = go ? S.c.t : S.c.tnext;
            while (iout < nout && t_out <= tacc) {
                if (special) emit(iout, M.y);
                if (W.i >= 0) rows(iout, W.i, W.y);
                iout++;
                if (iout < nout) t_out = tout[iout];
            }
        }
        if (!go) break;
        ok = row_step(tm, special, warp - 2, nrw, H, sl, P, D, k, S, S.pt[cur], M, B, W);
        // non-finite entries of the candidate, and of the step's start (state or d f / d a)
        if (W.i >= 0) {
            const double u = W.i == 0 ? M.u[0] : W.u;
            if (!xfinite(u + M.K[7 * n + W.i])) atomicAdd(&S.c.nbad_cand, 1);
            if (!(xfinite(W.y) && xfinite(W.col0))) atomicAdd(&S.c.nbad_start, 1);
        }
        bar_sync(1, c_rows);
    }
    if (R.status == DISCOEB_OK && iout < nout) R.status = DISCOEB_MAX_STEPS;
    R.outputs = iout;
    return R;
}

}  // namespace blk
}  // namespace dscb

#endif
