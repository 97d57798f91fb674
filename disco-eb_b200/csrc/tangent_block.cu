// Forward-mode solve on a block of warps per (mode, group of directions): kernel and launch.
#define DSCB_CALL_MATH
#include <cuda_runtime.h>

#include "discoeb.h"
#include "emit_output.cuh"
#include "tangent_block.cuh"
#include "tangent_block_launch.cuh"

using namespace dscb;

namespace {

constexpr int kMaxThreads = 512;

// Warps: the forward solve's (solve_block.cuh), nd directions, two producers of sources.  The step
// sequence is the forward's only: the tangent is the derivative of the discrete solution with its
// accepted steps held fixed.  Every wait between the three groups is bounded (handover.cuh); if one
// gives up, all of them leave and the mode reports DISCOEB_ABORTED.
//
// Gated: leaves if the older kernel's form has the launch (asked in every instantiation, it costs 1 to 3%).
template <bool Full, bool Gated>
__global__ void __launch_bounds__(kMaxThreads, 1) jvp_warps_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo,
    const DiscoebTangent* __restrict__ tangents, int n_dir, int nd_max, Dims D0, DiscoebControl ctrl, int n_modes,
    const double* __restrict__ kmodes, const double* __restrict__ tau_start, const double* __restrict__ y0,
    const double* __restrict__ y0_dot, const double* __restrict__ sw, int n_out, const double* __restrict__ tau_out,
    const double* __restrict__ tau_out_dot, double* y_out, double* y_out_dot, int32_t* status, int32_t* nsteps,
    int gate)
{
    extern __shared__ double smem[];
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int warp = threadIdx.x >> 5;
    const int groups = (n_dir + nd_max - 1) / nd_max;
    const int mode = blockIdx.x / groups, grp = blockIdx.x - mode * groups;
    const int d0 = grp * nd_max, nd = min(nd_max, n_dir - d0);
    if constexpr (Gated)
        if (!short_chain_wins(tm, n_modes, kmodes, n_out, gate)) {
            if (threadIdx.x == 0 && grp == 0) status[mode] = kOtherForm;
            return;
        }
    const int W = Full ? D0.n : 20;
    const double qnan = __longlong_as_double(0x7ff8000000000000LL);
    DiscoebCosmo* P = reinterpret_cast<DiscoebCosmo*>(smem);
    const blk::TanLayout L = blk::tan_layout(D0, nd_max);
    DiscoebTangent* TN = reinterpret_cast<DiscoebTangent*>(smem + L.tans);
    blk::Shared& S = *reinterpret_cast<blk::Shared*>(smem + L.shared);
    const blk::RowTable rows(smem + L.rows, L.nh);
    volatile int* flags = reinterpret_cast<int*>(smem + L.flags);
    const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
    bool bad = ci < 0 || ci >= n_cosmo;  // invalid cosmology index: report, solve nothing
    if (!bad) {
        const int* src = reinterpret_cast<const int*>(cosmos + ci);
        for (int i = threadIdx.x; i < (int)(sizeof(DiscoebCosmo) / 4); i += blockDim.x) reinterpret_cast<int*>(P)[i] = src[i];
        const int* ts = reinterpret_cast<const int*>(tangents + (size_t)ci * n_dir + d0);
        for (int i = threadIdx.x; i < nd * (int)(sizeof(DiscoebTangent) / 4); i += blockDim.x)
            reinterpret_cast<int*>(TN)[i] = ts[i];
        for (int i = threadIdx.x; i < nd_max * L.work_size; i += blockDim.x) smem[L.work + i] = 0.0;
        if (threadIdx.x < blk::kTanFlags) flags[threadIdx.x] = 0;
    }
    __syncthreads();
    Dims D{};
    if (!bad) {
        D = make_dims(*P);
        bad = !same_layout(D, D0);
    }
    if (bad) {  // (every cosmology must have the sizes of the first)
        if (threadIdx.x == 0 && grp == 0) {
            status[mode] = DISCOEB_BAD_INDEX;
            nsteps[mode] = 0;
        }
        for (int dd = 0; dd < nd; ++dd)
            for (int i = threadIdx.x; i < n_out * W; i += blockDim.x) {
                y_out_dot[((size_t)(d0 + dd) * n_modes + mode) * n_out * W + i] = qnan;
                if (d0 + dd == 0 && y_out) y_out[(size_t)mode * n_out * W + i] = qnan;
            }
        return;
    }
    const int n = D.n, forward = blk::row_warps(D) + 4;
    const double k = kmodes[mode];
    const double* tout = tau_out + (size_t)ci * n_out;
    const ModeMem M = blk::block_carve(smem + L.fwd, D);
    {
        const blk::Bands B = blk::make_bands(D, M.A);
        for (int hh = threadIdx.x; hh < L.nh; hh += blockDim.x) blk::fill_row(*P, D, B, k, hh, rows);
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) M.y[i] = y0[(size_t)mode * n + i];
    __syncthreads();
    const long long budget = poll_budget(ctrl);
    if (warp < forward) {
        const double swm[3] = {sw[3 * mode], sw[3 * mode + 1], sw[3 * mode + 2]};
        int cur = 0;  // which of S.pt the step started from
        auto accept = [&](double t, double h, double tnext, int regime) -> bool {
            const int m = flags[blk::FL_TOTAL], sl = m & 1;
            if (m >= 2 && !wait_at_least(tm, flags + blk::FL_CONSUMED + sl, nd * (m / 2), flags + blk::FL_ABORT, budget))
                return false;
            double* s = smem + L.slot + sl * L.slot_size;
            double* sc = s + L.sc;
            if (tm.lane < 8) s[L.K + tm.lane * n] = M.K[tm.lane * n];
            if (tm.leader()) {
                const blk::Point& pt = S.pt[cur];
                sc[blk::SL_ETAC] = pt.etac;
                for (int j = 0; j < 3; ++j) sc[blk::SL_F1 + j] = pt.f1u[j];
                sc[blk::SL_AL2] = S.c.al2;
                sc[blk::SL_AU2] = S.c.au2;
                sc[blk::SL_T] = t;
                sc[blk::SL_H] = h;
                sc[blk::SL_TNEXT] = tnext;
                sc[blk::SL_REGIME] = (double)regime;
            }
            tm.sync();
            cur ^= 1;
            return true;
        };
        auto emit = [](int, const double*) {};
        auto rows_out = [](int, int, double) {};
        const blk::StepPublisher publish{smem + L.slot, flags, L};
        const SolveResult R = blk::solve_mode_block(*P, D, ctrl, k, tau_start[mode], swm, n_out, tout, M, S, emit,
                                                    rows_out, accept, publish);
        if (warp == 0) {
            if (tm.leader()) {
                __threadfence_block();
                flags[blk::FL_DONE] = 1;
                if (grp == 0) nsteps[mode] = R.steps;
            }
            tm.sync();
            report_status(tm, R.status, flags[blk::FL_TOTAL], 2, nd, flags + blk::FL_CONSUMED, flags + blk::FL_ABORT,
                          budget, groups > 1, status + mode);
        }
        return;
    }
    if (warp >= forward + nd_max) {  // producers
        const int pw = warp - forward - nd_max;
        int hint = P->xe_loga.n_knots / 2;
        for (int m = 0;; ++m) {
            const int sl = m & 1;
            if (pw == 0) {
                if (tm.leader()) {
                    int have = 0;
                    long long polls = 0;
                    while (true) {
                        if (flags[blk::FL_PUBLISHED + sl] == m + 1) { have = 1; break; }
                        if (flags[blk::FL_DONE] && flags[blk::FL_TOTAL] <= m) break;
                        if (flags[blk::FL_ABORT]) break;
                        if (++polls > budget) { flags[blk::FL_ABORT] = 1; break; }
                        __nanosleep(100);
                    }
                    __threadfence_block();
                    flags[blk::FL_HAVE] = have;
                }
            }
            blk::bar_sync(blk::kBarProduce, 32 * blk::kProducers);
            if (!flags[blk::FL_HAVE]) break;
            blk::produce_step(tm, pw, *P, D, k, TN, nd, L, smem + L.slot + sl * L.slot_size, smem + L.base, hint);
            __threadfence_block();
            blk::bar_sync(blk::kBarProduce, 32 * blk::kProducers);
            if (pw == 0 && tm.leader()) flags[blk::FL_PRODUCED + sl] = m + 1;
        }
        return;
    }
    // ---- direction d0 + dl ----
    const int dl = warp - forward, dir = d0 + dl;
    if (dl >= nd) return;  // surplus warps of the last group
    double* w = smem + L.work + dl * L.work_size;
    double *yd = w + L.yd, *Kd = w + L.Kd;
    TanMem TT{};
    TT.yd = yd;
    TT.fd = Kd;  // (the stages' tangents are free between steps)
    TT.jk = Kd + n;
    double *pf = Kd + 2 * n, *yend = Kd + 3 * n;
    for (int i = tm.lane; i < n; i += 32) yd[i] = w[L.ud + i] = y0_dot[((size_t)dir * n_modes + mode) * n + i];
    tm.sync();
    const bool deferred = Full && y_out;
    int iout = 0;
    for (int m = 0;; ++m) {
        const int sl = m & 1;
        // one of them waits for all: they start each step together, and share its instruction fetches
        // (each waiting by itself, the steps took twice as long)
        if (dl == 0 && tm.leader()) {
            int have = 0;
            long long polls = 0;
            while (true) {
                if (flags[blk::FL_PRODUCED + sl] == m + 1) { have = 1; break; }
                if (flags[blk::FL_DONE] && flags[blk::FL_TOTAL] <= m) break;
                if (flags[blk::FL_ABORT]) break;
                if (++polls > budget) { flags[blk::FL_ABORT] = 1; break; }
                __nanosleep(100);
            }
            __threadfence_block();
            flags[blk::FL_HAVE_DIR] = have;
        }
        blk::bar_sync(blk::kBarDirect, 32 * nd);
        const int have = flags[blk::FL_HAVE_DIR];
        blk::bar_sync(blk::kBarDirect, 32 * nd);
        if (!have) break;
        const double* s = smem + L.slot + sl * L.slot_size;
        const double tnext = s[L.sc + blk::SL_TNEXT];
        const int regime = (int)s[L.sc + blk::SL_REGIME];
        blk::direction_step(tm, dl, D, k, L, nd, s, w, rows);
        bool out = iout < n_out && tout[iout] <= tnext;
        if (out)
            for (int i = tm.lane; i < n; i += 32) yend[i] = s[L.U + 6 * n + i] + s[L.K + 7 * n + i];
        tm.sync();
        if (tm.leader()) {
            __threadfence_block();
            atomicAdd(const_cast<int*>(flags) + blk::FL_CONSUMED + sl, 1);  // the slot may be overwritten from here on
        }
        tm.sync();
        while (deferred && iout < n_out && tout[iout] <= tnext) {  // as they are, for project_tangents_kernel
            const size_t oo = (size_t)mode * n_out + iout;
            for (int i = tm.lane; i < n; i += 32) {
                y_out_dot[((size_t)dir * n_modes * n_out + oo) * n + i] = yd[i];
                if (dir == 0) y_out[oo * n + i] = yend[i];
            }
            ++iout;
        }
        while (iout < n_out && tout[iout] <= tnext) {
            emit_tangent_output<Full>(tm, *P, TN + dl, D, k, mode, dir, n_modes, n_out, iout, tout,
                                      tau_out_dot + (size_t)ci * n_dir * n_out, yend, regime, TT, pf, y_out, y_out_dot);
            ++iout;
        }
        tm.sync();
        if (out)
            for (int i = tm.lane; i < 4 * n; i += 32) Kd[i] = 0.0;  // (zero times these enters the next sums)
        tm.sync();
    }
    for (int j = iout; j < n_out; ++j) {
        const size_t oo = (size_t)mode * n_out + j;
        for (int i = tm.lane; i < W; i += 32) {
            y_out_dot[((size_t)dir * n_modes * n_out + oo) * W + i] = qnan;
            if (dir == 0 && y_out) y_out[oo * W + i] = qnan;
        }
    }
}

// Whole states at the output times (emit_tangent_output's Full form) of a solve that stored states and
// tangents as they are: a block per (mode, output), warp 0 with the right-hand side at the output time
// (for the moving output time), then a warp per direction with the RSA projection.  In the solve this
// sat on the directions' chain of steps, 40 thousand cycles per output: 128 modes, 200 outputs, six
// directions 46 -> 28 ms.  Switch times are step boundaries, so the regime of the step that ended at an
// output follows from the times alone.
constexpr int kProjectWarps = 6;
__global__ void __launch_bounds__(32 * kProjectWarps) project_tangents_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo,
    const DiscoebTangent* __restrict__ tangents, int n_dir, Dims D0, int n_modes, const double* __restrict__ kmodes,
    const double* __restrict__ sw, int n_out, const double* __restrict__ tau_out, const double* __restrict__ tau_out_dot,
    const int32_t* __restrict__ status, double* y_out, double* y_out_dot)
{
    extern __shared__ double smem[];
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int warp = threadIdx.x >> 5, mode = blockIdx.x / n_out, j = blockIdx.x - mode * n_out;
    const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
    if (ci < 0 || ci >= n_cosmo) return;
    const DiscoebCosmo& P = cosmos[ci];
    const Dims D = make_dims(P);
    if (!same_layout(D, D0) || status[mode] == kOtherForm) return;
    const int n = D.n;
    double *y = smem, *f = y + n, *jk = f + n + warp * n;
    double* yo = y_out + ((size_t)mode * n_out + j) * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = yo[i];
    __syncthreads();
    if (!(y[0] == y[0])) return;  // never reached
    const double k = kmodes[mode], tau = tau_out[(size_t)ci * n_out + j];
    if (warp == 0) {
        const double* w = sw + 3 * (size_t)mode;
        const bool rsa = P.use_rsa && tau > w[0], ufa = !rsa && P.use_ufa && tau > w[1];
        int hint = P.xe_loga.n_knots / 2;
        Bg<double> b;
        bg_eval_team(tm, P, y[0], tau, k, (rsa ? 1 : 0) | (ufa ? 2 : 0), b, hint);
        rhs_team(tm, P, D, b, k, tau, y, f, (double*)nullptr);
    }
    __syncthreads();
    for (int d = warp; d < n_dir; d += kProjectWarps) {
        double* yd = y_out_dot + (((size_t)d * n_modes + mode) * n_out + j) * n;
        const double td = tau_out_dot[((size_t)ci * n_dir + d) * n_out + j];
        for (int i = tm.lane; i < n; i += 32) jk[i] = yd[i] + f[i] * td;
        tm.sync();
        Dual fld[4];
        const bool rsa = rsa_projection<Dual>(P, tangents + (size_t)ci * n_dir + d, D, tau, k, y, jk, fld);
        for (int i = tm.lane; i < n; i += 32) {
            double v = y[i], vd = jk[i];
            if (rsa) {
                const int sl = rsa_slot(D, i);
                if (sl >= 0) { v = fld[sl].v; vd = fld[sl].d; }
                else if (sl == -1) { v = 0.0; vd = 0.0; }
            }
            yd[i] = vd;
            if (d == 0) yo[i] = v;
        }
        tm.sync();
    }
}

}  // namespace

namespace dscb {
namespace blk {

int jvp_directions(const Dims& D, int want, size_t max_smem, size_t& smem)
{
    const int fixed = block_threads(D) + 32 * kProducers;
    int nd = want;
    while (nd > 0 && (fixed + 32 * nd > kMaxThreads || tan_layout(D, nd).total * sizeof(double) > max_smem)) --nd;
    if (nd == 0) return 0;
    const int groups = (want + nd - 1) / nd;  // even groups
    nd = (want + groups - 1) / groups;
    smem = tan_layout(D, nd).total * sizeof(double);
    return nd;
}

template <bool Full>
int32_t launch_jvp_block(const DiscoebCosmo* cosmos, int n_cosmo, const int32_t* mode_cosmo,
                         const DiscoebTangent* tangents, int n_dir, int nd, size_t smem, const Dims& D,
                         const DiscoebControl& ctrl, int n_modes, const double* kmodes, const double* tau_start,
                         const double* y0, const double* y0_dot, const double* sw, int n_out, const double* tau_out,
                         const double* tau_out_dot, double* y_out, double* y_out_dot, int32_t* status, int32_t* nsteps,
                         int gate, cudaStream_t stream)
{
    const auto kernel = gate != FormChoice::kOnly ? jvp_warps_kernel<Full, true> : jvp_warps_kernel<Full, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DISCOEB_ECUDA;
    const long long blocks = (long long)n_modes * ((n_dir + nd - 1) / nd);
    if (blocks > 0x7fffffffLL) return DISCOEB_EINVAL;
    if (blocks > n_modes && cudaMemsetAsync(status, 0, (size_t)n_modes * sizeof(int32_t), stream) != cudaSuccess)
        return DISCOEB_ECUDA;  // (several blocks report a mode: report_status)
    kernel<<<(unsigned)blocks, block_threads(D) + 32 * (nd + kProducers), smem, stream>>>(
        cosmos, n_cosmo, mode_cosmo, tangents, n_dir, nd, D, ctrl, n_modes, kmodes, tau_start, y0, y0_dot, sw, n_out,
        tau_out, tau_out_dot, y_out, y_out_dot, status, nsteps, gate);
    if (Full && y_out)
        project_tangents_kernel<<<(unsigned)((long long)n_modes * n_out), 32 * kProjectWarps,
                                  (2 + kProjectWarps) * D.n * sizeof(double), stream>>>(
            cosmos, n_cosmo, mode_cosmo, tangents, n_dir, D, n_modes, kmodes, sw, n_out, tau_out, tau_out_dot, status,
            y_out, y_out_dot);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}
template int32_t launch_jvp_block<false>(const DiscoebCosmo*, int, const int32_t*, const DiscoebTangent*, int, int,
                                         size_t, const Dims&, const DiscoebControl&, int, const double*, const double*,
                                         const double*, const double*, const double*, int, const double*, const double*,
                                         double*, double*, int32_t*, int32_t*, int, cudaStream_t);
template int32_t launch_jvp_block<true>(const DiscoebCosmo*, int, const int32_t*, const DiscoebTangent*, int, int,
                                        size_t, const Dims&, const DiscoebControl&, int, const double*, const double*,
                                        const double*, const double*, const double*, int, const double*, const double*,
                                        double*, double*, int32_t*, int32_t*, int, cudaStream_t);

}  // namespace blk
}  // namespace dscb
