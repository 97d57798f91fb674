// The tangents of a mode's accepted steps, six directions beside the forward solve (device only).
//
// A step's tangent along direction d obeys W K_s' = f'(u_s) + sum C_sj K_j' / h + h d_s f_t' + J' K_s
// (stepper.cuh, tangent_stage).  Rows >= 1 of f are linear in y[1:] with coefficients that depend on
// the scale factor a, on tau and on the parameters, so with c running over {a, theta_1, ...}
//
//   f'(u_s)  = L_s u_s' + a_s' (d_a L_s) u_s + (d_theta L_s) u_s
//   J' K_s   = y_0' (d_a L_0) K_s + (d_theta L_0) K_s
//              + K_s[0] (d_a L_0 y' + y_0' (d_a d_a L_0) y + (d_a d_theta L_0) y)
//
// where everything but L_s u_s' and d_a L_0 y' depends on the forward step alone.  That is where the
// dual numbers are, and they were the tangent's cost when each direction's warp evaluated its own:
// 206 us per step, nearly all of it scalar code that 32 lanes repeated.  Here two producer warps
// evaluate the sources of step m + 1, a lane per (stage, c), and tabulate L_s as functionals and row
// coefficients, while the directions' warps, one each, carry step m's tangents: plain FP64 sums, the
// chain substitutions with the forward's factors, and the rank-3 correction.
//
// Steps pass through two slots in shared memory: forward -> producers -> directions -> forward.
//
// What bounds it: instruction fetch.  Sixteen warps run through some 300 KB of code in every step;
// 41% of the instruction-cache requests miss, a miss per 16 cycles and SM, and "no instruction" is
// the first stall (5.6 of 12 cycles per issue).  Hence the tables instead of evaluated right-hand
// sides, one code path for all stages' sources, loops left rolled, and directions that start each
// step together.  512 modes to k = 10, 143 rows, six directions: 253 -> 139 ms; 48 modes 73 -> 28 ms;
// 80 modes of 219 rows 214 -> 63 ms.
#pragma once

#include "handover.cuh"
#include "solve_block.cuh"

#if defined(__CUDACC__)

namespace dscb {
namespace blk {

constexpr int kTan = (sizeof(DiscoebTangent) + 7) / 8;
constexpr int kProducers = 2;
constexpr int kSpec = 17;     // a source's special rows and its metric functionals h', eta'
constexpr int kBarProduce = 12, kBarDirect = 13;
enum { SL_CINV = 0, SL_F1 = 9, SL_ETAC = 12, SL_AL2, SL_AU2, SL_T, SL_H, SL_TNEXT, SL_REGIME, SL_SCALARS = 20 };
enum { FL_PUBLISHED = 0, FL_CONSUMED = 2, FL_DONE = 4, FL_TOTAL = 5, FL_ABORT = 6, FL_PRODUCED = 7, FL_HAVE = 9, FL_HAVE_DIR = 10,
       kTanFlags = 11 };

constexpr int kBgDual = sizeof(Bg<Dual>) / 8;

// The special rows' coefficients, in a table per stage that every lane reads through indices of its own:
// constants of the regime first, then what depends on the background.
enum { T_ZERO, T_ONE, T_MINUS, T_MHALF, T_M43, T_M23, T_K4, T_MK2, T_815, T_M6K, T_415, T_85, T_215, T_STATIC = 16,
       T_MAH = 16, T_R6LO, T_R6DI, T_R6U0, T_R6FAR, T_R6ETA, T_OPAC, T_MOPAC, T_OPAC10, T_R12DI, T_R13DI, T_R13UP,
       T_R13U0, T_R14LO, T_R14DI, T_F1U0, T_STAGE = 16 };

struct TanLayout {
    int n, nq, nh, ns, gs, nd, pc, ne;
    int tans, shared, fwd, rows, base, slot, slot_size, work, work_size, flags, total;  // doubles
    // within a slot
    int y, K, col0, U, G, sc, E, Z, F, H, sig, hsig, GT, dG, T, dT, vel, dvel;
    // within a direction's workspace
    int yd, ud, Kd, z, s0;
};
inline __host__ __device__ TanLayout tan_layout(const Dims& D, int nd)
{
    TanLayout L;
    const int n = D.n;
    L.n = n; L.nq = D.nq; L.nh = n_hier_rows(D); L.ns = n_slots(D); L.nd = nd; L.pc = positions_of(D); L.ne = 1 + D.nq;
    L.gs = 3 * L.ns > kBgDual ? 3 * L.ns : kBgDual;  // (a stage's background lies there until its functionals do)
    int o = 0;
    auto take = [&](int k) { const int at = o; o += k; return at; };
    L.y = take(n); L.K = take(8 * n); L.col0 = take(n); L.U = take(7 * n); L.G = take(4 * L.ns);
    L.sc = take(SL_SCALARS); L.E = take(3 * L.pc); L.Z = take(3 * L.pc);
    L.F = take(8 * (nd + 2) * kSpec); L.H = take((nd + 1) * kSpec);
    L.sig = take(8 * (nd + 1) * L.ne); L.hsig = take((nd + 1) * L.ne);
    L.GT = take(8 * L.gs); L.dG = take(3 * L.ns); L.T = take(T_STATIC + 8 * T_STAGE); L.dT = take(T_STATIC + T_STAGE);
    L.vel = take(8 * L.ne); L.dvel = take(L.ne);
    L.slot_size = o;
    o = 0;
    L.yd = take(n); L.ud = take(n); L.Kd = take(8 * n); L.z = take(L.pc); L.s0 = take(2 * kSpec + 3 * L.ne);
    L.work_size = o;
    o = 0;
    take(kCosmo);
    L.tans = take(nd * kTan); L.shared = take(kSharedDoubles); L.fwd = take(block_mem_doubles(D));
    L.rows = take(6 * L.nh); L.base = take((nd + 1) * (kBgDual + 4 * D.nq));
    L.work = take(nd * L.work_size); L.slot = take(2 * L.slot_size); L.flags = take((kTanFlags + 1) / 2);
    L.total = o + 4 * kWide;  // (the chains' look-ahead)
    return L;
}

// A hierarchy row's constants: k times its lower and upper coefficient (times the bin's velocity where
// massive), its couplings to h' and eta', L + 1 on the truncation row, and its indices
struct RowTable {
    double *lo, *up, *u0, *u1, *tr;
    uint2* at;
    __device__ __forceinline__ RowTable(double* p, int nh)
        : lo(p), up(p + nh), u0(p + 2 * nh), u1(p + 3 * nh), tr(p + 4 * nh), at(reinterpret_cast<uint2*>(p + 5 * nh))
    {
    }
};
enum { R_MASSIVE = 1u << 25, R_OPAQUE = 1u << 26, R_RSA0 = 1u << 27, R_UFA0 = 1u << 28, R_POL0 = 1u << 29, R_POL2 = 1u << 30 };
__device__ __forceinline__ void fill_row(const DiscoebCosmo& P, const Dims& D, const Bands& B, double k, int hh,
                                         const RowTable& R)
{
    const int i = hier_row(D, hh);
    int l, L, species;
    if (i <= 7 + D.lmaxg) { l = i - 7; L = D.lmaxg; species = 0; }
    else if (i <= D.idxgp + D.lmaxgp) { l = i - D.idxgp; L = D.lmaxgp; species = 1; }
    else if (i <= D.idxr + D.lmaxr) { l = i - D.idxr; L = D.lmaxr; species = 2; }
    else { l = div_nq(i - D.iq0, D.nq); L = D.lmaxnu; species = 3; }
    const bool massive = species == 3, trunc = l == L;
    const int st = massive ? D.nq : 1, q = hier_bin(D, i);
    const double io = inv_odd(l), dl = massive ? dlfdlq_of(P.q[q]) : 0.0;
    R.lo[hh] = trunc ? k : k * (l * io);
    R.up[hh] = trunc ? 0.0 : -k * ((l + 1.0) * io);
    R.u0[hh] = l == 0 ? dl * (1.0 / 6.0) : (l == 2 ? -dl * (1.0 / 15.0) : 0.0);
    R.u1[hh] = l == 2 ? -0.4 * dl : 0.0;
    R.tr[hh] = trunc ? L + 1.0 : 0.0;
    R.at[hh] = make_uint2((unsigned)i | (unsigned)position(D, B, i) << 16,
                          (unsigned)(i - st) | (unsigned)(trunc ? i : i + st) << 10 | (unsigned)(massive ? 1 + q : 0) << 20 |
                              (massive ? R_MASSIVE : 0u) | (species <= 1 ? R_OPAQUE : 0u) | (species <= 2 ? R_RSA0 : 0u) |
                              (species == 2 ? R_UFA0 : 0u) | (species == 1 && l == 0 ? R_POL0 : 0u) |
                              (species == 1 && l == 2 ? R_POL2 : 0u));
}

// products as the source writes them
struct PlainProducts {
    template <class A, class B> static __device__ __forceinline__ A product(const A& x, const B& y) { return x * y; }
    template <class T> static __device__ __forceinline__ T rsa_theta(const T& H, const T& fac, const T& Y)
    {
        return -0.5 * H + fac * Y;
    }
    template <class T> static __device__ __forceinline__ T rsa_inner(const T& a, double x, const T& b, double y, double c,
                                                                     double z)
    {
        return a * x + b * y + c * z;
    }
};
// special rows on one lane
template <class T, class IV>
__device__ __forceinline__ void special_lane(const DiscoebCosmo& P, const Dims& D, const Bg<T>& b, double k, double tau,
                                             const double* y, IV bins, T sp[15], T& g0, T& g1)
{
    T drho = 0.0, dp = 0.0, fnu = 0.0, g2;
    const double* yq = y + D.iq0;
#pragma unroll 1
    for (int q = 0; q < D.nq; ++q) {
        T iv, v;
        bins(q, iv, v);
        const double w = P.wq[q], wy = w * yq[q];
        drho = drho + wy * iv;
        dp = dp + wy * v;
        fnu = fnu + T(w * yq[D.nq + q]);
    }
    special_core<T, double, PlainProducts>(P, D, b, k, tau, StateAt{y}, drho, dp, fnu, sp, g0, g1, g2);
}

// ---- forward: the accepted steps into the slots ----
struct StepPublisher {
    double* slots;
    volatile int* flags;
    const TanLayout& L;
    __device__ __forceinline__ void copy(int i, double y, const ModeMem& M, const Bands& B, int tid, int nt) const
    {
        double* s = slots + (flags[FL_TOTAL] & 1) * L.slot_size;
        const int n = L.n;
        if (i >= 0) {
            s[L.y + i] = y;
            s[L.col0 + i] = M.col0[i];
            if (i >= 1)
#pragma unroll
                for (int j = 0; j < 8; ++j) s[L.K + j * n + i] = M.K[j * n + i];
        }
        for (int x = tid; x < L.pc; x += nt) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                s[L.E + 3 * x + j] = B.E[4 * x + j];
                s[L.Z + j * L.pc + x] = B.Z[j * L.pc + x];
            }
        }
        for (int x = tid; x < L.ns; x += nt) {
#pragma unroll
            for (int r = 0; r < 4; ++r) s[L.G + r * L.ns + x] = M.Gs[r * kMaxSlots + x];  // F1s follows
        }
        if (tid < 9) s[L.sc + SL_CINV + tid] = M.sc[SC_CINV + tid];
        if (tid >= 9 && tid < 12) s[L.sc + SL_F1 + tid - 9] += M.sc[SC_F1Z + tid - 9];  // f1u is there
    }
    __device__ __forceinline__ void done(const ModeMem&) const
    {
        if ((threadIdx.x & 31) == 0) {
            const int m = flags[FL_TOTAL];
            flags[FL_TOTAL] = m + 1;
            __threadfence_block();
            flags[FL_PUBLISHED + (m & 1)] = m + 1;
        }
        __syncwarp();
    }
};

// ---- producers: a step's sources ----
// bg_eval on one lane, the tables in a loop (the kernel is bound by instruction fetch)
template <class T>
__device__ __forceinline__ void lane_bg(const DiscoebCosmo& P, T a, double tau, double k, int regime, Bg<T>& b, int& hint,
                                        const DiscoebTangent* tn)
{
    const Par<T> par = make_par<T>(P, tn);
    const T loga = xlog(a);
    BgTables<T> tb;
#pragma unroll 1
    for (int t = 0; t < 5; ++t) {
        int i = 0;
        if (t < 4) i = table_slot_index(P, t, val(loga), hint);
        T slope, y = table_slot_eval(P, par, tn, t, i, a, loga, slope);
        if (t >= 2) y = xexp(y);
        if (t == 0) { tb.xe = y; tb.xep = slope; }
        else if (t == 1) tb.cs2a = y;
        else if (t == 2) tb.rhonu = y;
        else if (t == 3) tb.pnu = y;
        else tb.rho_Q = y;
    }
    bg_finish(P, par, a, tb, tau, k, regime, b);
}

// the functionals of stage q on the state slots (gcol, f1col), one lane
__device__ __forceinline__ void stage_functionals(const DiscoebCosmo& P, const Dims& D, const Bg<Dual>& b, double k,
                                                  const TanLayout& L, double* s, int q)
{
    const double k2 = k * k, sk2 = k2 > 1e-30 ? k2 : 1e-30, hE = 0.5 * rcp(k2), third = 1.0 / 3.0;
    const int nq = D.nq, ns = L.ns, de = 12 + 2 * nq;
    double *GT = s + L.GT + q * L.gs, *dG = s + L.dG;
    const bool rsa = b.rsa;
    const Dual ih = b.iaHG, ia2 = b.ia2, fac = b.rsa_fac, cg = (hE * (4.0 / 3.0) * P.grhog) * ia2;
    const Dual cr = (hE * (4.0 / 3.0) * P.Neff * P.grhor) * ia2;
    Dual eH = 0.0;
    if (rsa) eH = cg * (-0.5 - 0.5 * fac * b.rsa_tcs) - 0.5 * cr;
    auto set = [&](int x, int j, const Dual& v) {
        GT[x * ns + j] = v.v;
        if (q == 0) dG[x * ns + j] = v.d;
    };
    // slot j: the density's and momentum's coefficients, and that of rho + 3 p
    auto put = [&](int j, const Dual& rho, const Dual& g1, const Dual& f) {
        const Dual g0 = rho * ih;
        set(0, j, g0);
        set(1, j, g1 + eH * g0);
        set(2, j, -b.a * f);
    };
    const Dual zero = 0.0, pg = P.grhog * ia2, pr = (P.grhor * P.Neff) * ia2;
    const Dual mc = b.par.grhom * (b.par.Omegam - b.par.Omegab) * b.ia, mb = b.par.grhom * b.par.Omegab * b.ia;
    const Dual dq = b.par.grhom * b.par.OmegaDE * b.rho_Q * b.a2;
    put(0, Dual(2.0 * k2), rsa ? cg * fac * sk2 : zero, rsa ? -4.0 * (pg + pr) : zero);
    put(1, mc, zero, mc);
    set(1, 2, hE * mc);
    put(3, mb, rsa ? cg * fac * (b.cs2 * sk2) : zero, mb);
    set(1, 4, rsa ? hE * mb + cg * fac * (-b.rsa_tcs - b.aH) : hE * mb);
    if (rsa) {
        set(2, 4, -b.a * (pg * ((4.0 / sk2) * (fac * (sk2 * third)))));
        set(2, 5, -b.a * pg);
        set(2, 10, -b.a * pr);
    } else {
        put(5, pg, zero, 2.0 * pg);
        set(1, 6, cg);
        put(10, pr, zero, 2.0 * pr);
        set(1, 11, cr);
    }
    put(de, dq, zero, (1.0 + 3.0 * P.cs2_DE) * dq);
    const Dual tq = b.opw * dq;
    set(1, de + 1, hE * tq);
    set(2, de + 1, -b.a * (3.0 * ((P.cs2_DE - b.ca2_Q) * (3.0 * b.aH * tq * rcp(k2)))));
    const double* vel = s + L.vel + q * L.ne;
#pragma unroll 1
    for (int j = 0; j < nq; ++j) {
        const Dual v(vel[1 + j], q == 0 ? s[L.dvel + 1 + j] : 0.0), w = (P.grhor * P.Nmnu * P.wq[j]) * ia2, rho = w * rcp(v);
        put(12 + j, rho, zero, rho + w * v);
        set(1, 12 + nq + j, (hE * k) * w);
    }
}
// what depends on the background in the special rows: T (values) and dT (d/da, may be null)
__device__ __forceinline__ void stage_rows(const DiscoebCosmo& P, const Bg<Dual>& b, double k, double* T, double* dT)
{
    const double k2 = k * k, sk2 = k2 > 1e-30 ? k2 : 1e-30, ik2 = rcp(k2), cs2Q = P.cs2_DE;
    auto put = [&](int i, const Dual& x) {
        T[i - T_STATIC] = x.v;
        if (dT) dT[i - T_STATIC] = x.d;
    };
    const Dual lo = k2 * b.cs2, di = -b.aH - b.po;
    put(T_MAH, -b.aH);
    put(T_OPAC, b.opac);
    put(T_MOPAC, -b.opac);
    put(T_OPAC10, 0.1 * b.opac);
    put(T_R12DI, Dual(-1.5 * b.itau));
    Dual f1[3];
    f1u<Dual>(P, b, k, f1);
    put(T_F1U0, f1[0]);
    if (b.rsa) {
        const Dual pf = b.po * b.rsa_fac;
        put(T_R6LO, lo + pf * (b.cs2 * sk2));
        put(T_R6DI, di + pf * (-b.rsa_tcs - b.aH));
        put(T_R6U0, b.po * (-0.5 - 0.5 * b.rsa_fac * b.rsa_tcs));
        put(T_R6ETA, pf * sk2);
        put(T_R6FAR, Dual(0.0));
    } else {
        put(T_R6LO, lo);
        put(T_R6DI, di);
        put(T_R6U0, Dual(0.0));
        put(T_R6ETA, Dual(0.0));
        put(T_R6FAR, b.po);
    }
    const double live = b.de_frozen ? 0.0 : 1.0;
    put(T_R13DI, (-3.0 * live) * ((cs2Q - b.w_Q) * b.aH));
    put(T_R13UP, live * (-b.opw - (9.0 * ik2) * (b.opw * (cs2Q - b.ca2_Q) * b.aH * b.aH)));
    put(T_R13U0, (-0.5 * live) * b.opw);
    put(T_R14LO, (cs2Q * k2 * live) * b.iopw);
    put(T_R14DI, (-(1.0 - 3.0 * cs2Q) * live) * b.aH);
}
// lane j's indices into that table: lower, main, upper diagonal, far column, eta, and h', eta', polter
struct SpecialIdx {
    unsigned a, b;  // four bytes each
};
__device__ __forceinline__ SpecialIdx special_idx(int j, bool rsa, bool ufa)
{
    int lo = 0, di = 0, up = 0, far = 0, eta = 0, u0 = 0, u1 = 0, u2 = 0;
    if (j == 2) u1 = T_ONE;
    else if (j == 3 || j == 5) { up = T_MINUS; u0 = T_MHALF; }
    else if (j == 4) di = T_MAH;
    else if (j == 6) { lo = T_R6LO; di = T_R6DI; far = T_R6FAR; u0 = T_R6U0; eta = T_R6ETA; }
    else if (j == 13) { di = T_R13DI; up = T_R13UP; u0 = T_R13U0; }
    else if (j == 14) { lo = T_R14LO; di = T_R14DI; }
    else if (rsa) {}
    else if (j == 7 || j == 10) { up = T_M43; u0 = T_M23; }
    else if (j == 8) { lo = T_K4; di = T_MOPAC; up = T_MK2; far = T_OPAC; }
    else if (j == 11) { lo = T_K4; up = T_MK2; }
    else if (j == 9) { lo = T_815; di = T_MOPAC; up = T_M6K; u0 = T_415; u1 = T_85; u2 = T_OPAC10; }
    else if (j == 12 && ufa) { lo = T_415; di = T_R12DI; u0 = T_215; }
    else if (j == 12) { lo = T_815; up = T_M6K; u0 = T_415; u1 = T_85; }
    return SpecialIdx{(unsigned)(lo | di << 8 | up << 16 | far << 24), (unsigned)(eta | u0 << 8 | u1 << 16 | u2 << 24)};
}

__device__ __forceinline__ void produce_step(const WarpTeam& tm, int pw, const DiscoebCosmo& P, const Dims& D, double k,
                                             const DiscoebTangent* TN, int nd, const TanLayout& L, double* s,
                                             double* base, int& hint)
{
    const int n = L.n, nq = L.nq, nc = nd + 1, tid = 32 * pw + tm.lane;
    const double t = s[L.sc + SL_T], h = s[L.sc + SL_H];
    const int regime = (int)s[L.sc + SL_REGIME];
    double *K = s + L.K, *U = s + L.U;
    // the stage states
    for (int i = tid; i < n; i += 32 * kProducers) {
        double kk[8], u = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) kk[j] = K[j * n + i];
        const double y = s[L.y + i];
#pragma unroll
        for (int q = 1; q < 8; ++q) {
            if (q <= 5) {
                u = y;
#pragma unroll
                for (int j = 0; j < 5; ++j)
                    if (j < q) u += kR5.a[q][j] * kk[j];
            } else {
                u += kk[q - 1];
            }
            U[(q - 1) * n + i] = u;
        }
    }
    bar_sync(kBarProduce, 32 * kProducers);
    // (stage q, component c)'s place among the sources: F of a, (J of a), the directions' sums
    auto place = [&](int q, int c) { return s + L.F + (q * (nc + 1) + (c == 0 ? 0 : 1 + c)) * kSpec; };
    // every stage in the numbers the step start needs (hyper-dual: along c, and along a): one code path
    for (int x = tid; x < 8 * nc; x += 32 * kProducers) {
        const int q = x / nc, c = x - q * nc;
        const double* u = q ? U + (q - 1) * n : s + L.y;
        const double ts = q <= 5 ? t + kR5.c[q] * h : t + h;
        Bg<HDual> b;
        lane_bg(P, HDual(Dual(u[0], c == 0 ? 1.0 : 0.0), Dual(1.0, 0.0)), ts, k, regime, b, hint, c ? TN + c - 1 : nullptr);
        double* sig = s + L.sig + (q * nc + c) * L.ne;
        double* hsig = s + L.hsig + c * L.ne;
        double* mine = base + c * (kBgDual + 4 * nq);
        double* vel = s + L.vel + q * L.ne;
        sig[0] = b.opac.v.d;
        if (c == 0) {
            vel[0] = 1.0;
            *reinterpret_cast<Bg<Dual>*>(s + L.GT + q * L.gs) = bg_value(b);
        }
        if (q == 0) {
            hsig[0] = b.opac.d.d;
            *reinterpret_cast<Bg<Dual>*>(mine) = bg_value(b);
        }
        Dual* d = reinterpret_cast<Dual*>(mine + kBgDual);
        auto bins = [&](int j, HDual& iv, HDual& v) {
            iv = inv_vq(P, b, j);
            v = rcp(iv);
            sig[1 + j] = v.v.d;
            if (c == 0) vel[1 + j] = v.v.v;
            if (q == 0) {
                hsig[1 + j] = v.d.d;
                if (c == 0) s[L.dvel + 1 + j] = v.v.d;
                d[j] = iv.v;
                d[nq + j] = v.v;
            }
        };
        HDual sp[15], g0, g1;
        special_lane<HDual>(P, D, b, k, ts, u, bins, sp, g0, g1);
        double* f = place(q, c);
#pragma unroll
        for (int j = 0; j < 15; ++j) f[j] = sp[j].v.d;
        f[15] = g0.v.d;
        f[16] = g1.v.d;
        if (q == 0) {
            double* hh = s + L.H + c * kSpec;
#pragma unroll
            for (int j = 0; j < 15; ++j) hh[j] = sp[j].d.d;
            hh[15] = g0.d.d;
            hh[16] = g1.d.d;
        }
    }
    bar_sync(kBarProduce, 32 * kProducers);
    // (d_c L_0) K_q: row 0 does not depend on the rows of K
    for (int x = tid; x < 8 * nc; x += 32 * kProducers) {
        const int q = x / nc, c = x - q * nc;
        const double* mine = base + c * (kBgDual + 4 * nq);
        const Bg<Dual>& b = *reinterpret_cast<const Bg<Dual>*>(mine);
        const Dual* d = reinterpret_cast<const Dual*>(mine + kBgDual);
        auto bins = [&](int j, Dual& iv, Dual& v) {
            iv = d[j];
            v = d[nq + j];
        };
        Dual sp[15], g0, g1;
        special_lane<Dual>(P, D, b, k, t, K + q * n, bins, sp, g0, g1);
        sp[0] = 0.0;
        if (c == 0) {
            double* f = place(q, 0) + kSpec;
#pragma unroll
            for (int j = 0; j < 15; ++j) f[j] = sp[j].d;
            f[15] = g0.d;
            f[16] = g1.d;
        } else {
            double* f = place(q, c);
#pragma unroll
            for (int j = 0; j < 15; ++j) f[j] += sp[j].d;
            f[15] += g0.d;
            f[16] += g1.d;
        }
    }
    // the stages' functionals and special rows (point_functionals, point_rows)
    if (pw == 0 && tm.lane < T_STATIC) {
        const double k2 = k * k, v[T_STATIC] = {0.0, 1.0, -1.0, -0.5, -4.0 / 3.0, -2.0 / 3.0, 0.25 * k2, -0.5 * k2,
                                                8.0 / 15.0, -0.6 * k, 4.0 / 15.0, 8.0 / 5.0, 2.0 / 15.0, 0.0, 0.0, 0.0};
        double x = 0.0;
#pragma unroll
        for (int j = 0; j < T_STATIC; ++j)
            if (j == tm.lane) x = v[j];
        s[L.T + tm.lane] = x;
        s[L.dT + tm.lane] = 0.0;
        if (tm.lane == 0) s[L.dvel] = 0.0;
    }
    if (pw == 1) {
        const int q = tm.lane < 8 ? tm.lane : 0;
        const Bg<Dual> b = *reinterpret_cast<const Bg<Dual>*>(s + L.GT + q * L.gs);
        tm.sync();
        for (int x = tm.lane; x < 8 * L.gs; x += 32) s[L.GT + x] = 0.0;
        for (int x = tm.lane; x < 3 * L.ns; x += 32) s[L.dG + x] = 0.0;
        tm.sync();
        if (tm.lane < 8) {
            stage_functionals(P, D, b, k, L, s, q);
            stage_rows(P, b, k, s + L.T + T_STATIC + q * T_STAGE, q == 0 ? s + L.dT + T_STATIC : nullptr);
        }
    }
}

// ---- one direction: a step's tangent ----
__device__ __forceinline__ void direction_step(const WarpTeam& tm, int dl, const Dims& D, double k, const TanLayout& L,
                                               int nd, const double* s, double* w, const RowTable& rows)
{
    const int n = L.n, nq = L.nq, nc = nd + 1, lane = tm.lane, ne = L.ne, ns = L.ns;
    const double *sc = s + L.sc, *K = s + L.K, *U = s + L.U, *col0 = s + L.col0, *Z = s + L.Z, *T = s + L.T;
    double *yd = w + L.yd, *ud = w + L.ud, *Kd = w + L.Kd, *z = w + L.z;
    double *src = w + L.s0, *hsrc = src + kSpec, *sg = hsrc + kSpec, *sg0 = sg + ne, *sgh = sg0 + ne;
    double* c0d = Kd + 7 * n;  // d/de (d f / d a); K_7' takes its place
    const double t = sc[SL_T], h = sc[SL_H], gh = kR5.gamma * h, ih = rcp(h), it2 = rcp(t * t);
    const int regime = (int)sc[SL_REGIME];
    const bool rsa = (regime & 1) != 0, ufa = !rsa && (regime & 2) != 0;
    const unsigned off = (rsa ? R_RSA0 : 0u) | (ufa ? R_UFA0 : 0u);  // species that stand still
    const double y0d = yd[0];
    const double iw00 = rcp(rcp(gh) - s[L.F]);  // (the a-derivative of f_0 is the first source)
    const Bands B = make_bands(D, const_cast<double*>(s + L.E));
    const Slots sl = make_slots(D, B, lane);
    const Slots su{lane < ns ? slot_index(D, lane) : 0, lane + 32 < ns ? slot_index(D, lane + 32) : 0, ns};
    auto load_g = [&](const double* g, int r0, int r1, int r3, double polter) {  // rows of ns; r2 is polter's
        SlotG G;
        const bool in = lane < ns, in2 = lane + 32 < ns;
        G.g[0] = in ? g[r0 * ns + lane] : 0.0;
        G.g[1] = in ? g[r1 * ns + lane] : 0.0;
        G.g[2] = polter;
        G.g[3] = in ? g[r3 * ns + lane] : 0.0;
        G.h[0] = in2 ? g[r0 * ns + lane + 32] : 0.0;
        G.h[1] = in2 ? g[r1 * ns + lane + 32] : 0.0;
        G.h[2] = 0.0;
        G.h[3] = in2 ? g[r3 * ns + lane + 32] : 0.0;
        return G;
    };
    const double pol = (!rsa && lane >= 7 && lane <= 9) ? 1.0 : 0.0;
    const SlotG G = load_g(s + L.G, 0, 1, 3, pol);
    const int si = lane < 15 ? special_row(D, lane) : -1;
    const int spos = si >= 1 ? position(D, B, si) : B.steps * B.nl, s1 = si >= 1 ? si : 1;
    const int sfar = lane == 6 ? 8 : 6;
    const SpecialIdx ix = special_idx(lane, rsa, ufa);
    const double f1z0 = sc[SL_F1], f1z1 = sc[SL_F1 + 1], f1z2 = sc[SL_F1 + 2];
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        const double* us = q ? U + (q - 1) * n : s + L.y;
        const double* Kq = K + q * n;
        const double ad = ud[0], K0 = Kq[0];
        const double* vel = s + L.vel + q * ne;
        const double opac = T[T_OPAC + q * T_STAGE], its = rcp(q <= 5 ? t + kR5.c[q] * h : t + h);
        double g[4];
        slot_sums<1>(tm, su, load_g(s + L.GT + q * L.gs, 0, 1, 2, pol), ud, g);
        auto at = [&](unsigned i) { return T[i + (i >= T_STATIC ? q * T_STAGE : 0)]; };
        // special rows: L_q u'
        double f = at(ix.a & 255u) * ud[s1 - 1] + at((ix.a >> 8) & 255u) * ud[s1] + at((ix.a >> 16) & 255u) * ud[s1 + 1];
        f += at(ix.a >> 24) * ud[sfar] + at(ix.b & 255u) * ud[2];
        f += at((ix.b >> 8) & 255u) * g[0] + at((ix.b >> 16) & 255u) * g[1] + at(ix.b >> 24) * g[2];
        if (lane == 1) f = g[3] + T[T_F1U0 + q * T_STAGE] * g[0];
        double gd[4] = {0.0, 0.0, 0.0, 0.0}, dopac = 0.0;
        if (q == 0) {
            // once per step, for every stage: d/de (d f / d a) of the special rows
            const double* dT = s + L.dT;
            slot_sums<1>(tm, su, load_g(s + L.dG, 0, 1, 2, 0.0), ud, gd);
            dopac = dT[T_OPAC];
            double fd = dT[ix.a & 255u] * ud[s1 - 1] + dT[(ix.a >> 8) & 255u] * ud[s1] + dT[(ix.a >> 16) & 255u] * ud[s1 + 1];
            fd += dT[ix.a >> 24] * ud[sfar] + dT[ix.b & 255u] * ud[2];
            fd += at((ix.b >> 8) & 255u) * gd[0] + at((ix.b >> 16) & 255u) * gd[1];
            fd += dT[(ix.b >> 8) & 255u] * g[0] + dT[ix.b >> 24] * g[2];
            if (lane == 1) fd = gd[3] + T[T_F1U0] * gd[0] + dT[T_F1U0] * g[0];
            if (lane == 0) fd = 0.0;
            if (lane < kSpec) {
                const double* H = s + L.H + lane;
                const double v = H[0] * y0d + H[(1 + dl) * kSpec];
                if (lane < 15) c0d[si] = fd + v;
                else hsrc[lane] = v;
            }
            if (lane < ne) {
                const double* a = s + L.sig + lane;
                const double* b = s + L.hsig + lane;
                sg0[lane] = a[0] * y0d + a[(1 + dl) * ne];
                sgh[lane] = b[0] * y0d + b[(1 + dl) * ne];
            }
        }
        // the stage's sources along this direction
        if (lane < kSpec) {
            const double* F = s + L.F + q * (nc + 1) * kSpec + lane;
            src[lane] = F[0] * ad + F[kSpec] * y0d + F[(2 + dl) * kSpec];
        }
        if (lane < ne) {
            const double* a = s + L.sig + q * nc * ne + lane;
            sg[lane] = a[0] * ad + a[(1 + dl) * ne];
        }
        tm.sync();
        double cc[7], ca[6];
#pragma unroll
        for (int j = 0; j < 7; ++j) cc[j] = kR5.C[q][j] * ih;
        const double hd = q < 5 ? h * kR5.d[q] : 0.0;
        auto stages = [&](int i) {
            double r0 = 0.0, r1 = 0.0;
#pragma unroll
            for (int j = 0; j < 6; j += 2) {
                r0 += cc[j] * Kd[j * n + i];
                r1 += cc[j + 1] * Kd[(j + 1) * n + i];
            }
            return (r0 + cc[6] * Kd[6 * n + i]) + r1;
        };
        const double x0 = (src[0] + K0 * c0d[0] + stages(0)) * iw00;
        {
            double v = 0.0;
            if (si >= 1) {
                v = f + src[lane] + K0 * c0d[si] + stages(si);
                if (lane == 12 && ufa && t > 1e-30) v += hd * (1.5 * it2 * yd[si]);
                v += col0[si] * x0;
            }
            if (si == 2) v *= gh;
            const double v2 = tm.bcast(v, 2);
            if (si == 6) v += sc[SL_ETAC] * v2;
            if (si >= 1) z[spos] = v;
        }
        // hierarchy rows
        const double pu = rsa ? 0.0 : us[9] + us[D.idxgp] + us[D.idxgp + 2];
        const double pk = rsa ? 0.0 : Kq[9] + Kq[D.idxgp] + Kq[D.idxgp + 2];
        const double e0 = g[0] + src[15], e1 = g[1] + src[16];
#pragma unroll 1
        for (int hh = lane; hh < L.nh; hh += 32) {
            const uint2 r = rows.at[hh];
            const int i = r.x & 0xffffu, im = r.y & 1023u, ip = (r.y >> 10) & 1023u, e = (r.y >> 20) & 31u;
            const bool on = (r.y & off) == 0, opaque = on && (r.y & R_OPAQUE), massive = (r.y & R_MASSIVE) != 0;
            const double lo = on ? rows.lo[hh] : 0.0, up = on ? rows.up[hh] : 0.0, tr = on ? rows.tr[hh] : 0.0;
            const double u0 = rows.u0[hh], u1 = rows.u1[hh], c2 = (r.y & R_POL0) ? 0.5 : ((r.y & R_POL2) ? 0.1 : 0.0);
            const double ui = ud[i], lin = lo * ud[im] + up * ud[ip];
            // sources: the bins' velocities and the opacity along the direction, at the stage and at the start
            const double lu = lo * us[im] + up * us[ip], lk = lo * Kq[im] + up * Kq[ip];
            const double qu = c2 * pu - us[i], qk = c2 * pk - Kq[i];
            const double xu = massive ? lu : qu, xk = massive ? lk : qk;
            const bool any = massive || opaque;
            const double sx = any ? sg[e] : 0.0, sx0 = any ? sg0[e] : 0.0;
            if (q == 0) {
                double d = lin * s[L.dvel + e] + u0 * (gd[0] + hsrc[15]) + u1 * (gd[1] + hsrc[16]);
                if (opaque) d += dopac * (c2 * g[2] - ui);
                c0d[i] = d + (any ? xu * sgh[e] : 0.0);
            }
            double v = lin * vel[e] - tr * (its * ui - hd * it2 * yd[i]);
            if (opaque) v += opac * (c2 * g[2] - ui);
            v += u0 * e0 + u1 * e1 + K0 * c0d[i];
            z[r.x >> 16] = v + (xu * sx + xk * sx0) + stages(i) + col0[i] * x0;
        }
        tm.sync();
        solve_short<1, 3>(B, lane, z, 1);
        if (lane < 3 + nq) solve_tri<1, 3>(B, lane, sc[SL_AL2], sc[SL_AU2], z);
        tm.sync();
        double gz[4];
        slot_sums<1>(tm, sl, G, z, gz);
        const double c0 = sc[0] * gz[0] + sc[1] * gz[1] + sc[2] * gz[2];
        const double c1 = sc[3] * gz[0] + sc[4] * gz[1] + sc[5] * gz[2];
        const double c2 = sc[6] * gz[0] + sc[7] * gz[1] + sc[8] * gz[2];
        double* Kn = Kd + q * n;
        // K_q', and with it the next stage's state (after the last, the step's)
#pragma unroll
        for (int j = 0; j < 5; ++j) ca[j] = q < 5 ? kR5.a[q + 1][j] : 0.0;
        const double cl = q < 5 ? kR5.a[q + 1][q] : 1.0;
        auto advance = [&](int i, double kv) {
            Kn[i] = kv;
            double v = (q < 5 ? yd[i] : ud[i]) + cl * kv;
            if (q < 5) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j < q) v += ca[j] * Kd[j * n + i];
            }
            ud[i] = v;
            if (q == 7) yd[i] = v;
        };
        if (si >= 0) {
            double kv = x0;
            if (si == 1) kv = gh * (z[spos] + gz[3] + (f1z0 * c0 + f1z1 * c1 + f1z2 * c2));
            else if (si > 1) kv = z[spos] + (Z[spos] * c0 + Z[L.pc + spos] * c1 + Z[2 * L.pc + spos] * c2);
            advance(si, kv);
        }
#pragma unroll 2
        for (int hh = lane; hh < L.nh; hh += 32) {
            const unsigned r = rows.at[hh].x, p = r >> 16;
            advance(r & 0xffffu, z[p] + (Z[p] * c0 + Z[L.pc + p] * c1 + Z[2 * L.pc + p] * c2));
        }
        tm.sync();
    }
}

}  // namespace blk
}  // namespace dscb

#endif
