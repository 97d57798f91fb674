// Forward perturbation solve on sm_100a: kernels and the C ABI (include/discoeb.h).
//
// The FP64 solves run on a block of warps per mode (solve_block.cu, tangent_block.cu) wherever that is
// the faster form; the kernels here take the rest.
//
// Layout of those: one warp owns one k-mode.  Its whole working set (state, eight Rodas5 stage
// vectors, the banded chain factors and the Woodbury blocks, 27 n doubles) lives in
// shared memory; the four background tables are read through the read-only cache.
// All modes of all cosmologies run in one launch; each warp takes modes from a
// grid-stride schedule ordered by the caller (longest first).  HBM traffic is only the
// initial states and the outputs, so the kernel is bound by FP64 latency, not bandwidth.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "discoeb.h"
#include "emit_output.cuh"
#include "handover.cuh"
#include "solve_block_launch.cuh"
#include "stepper.cuh"
#include "tangent_block_launch.cuh"

using namespace dscb;

namespace {

constexpr int kCosmoDoubles = (sizeof(DiscoebCosmo) + 7) / 8;

__device__ __forceinline__ void copy_cosmo(const WarpTeam& tm, const DiscoebCosmo* src, DiscoebCosmo* dst)
{
    const int* s = reinterpret_cast<const int*>(src);
    int* d = reinterpret_cast<int*>(dst);
    for (int i = tm.lane; i < (int)(sizeof(DiscoebCosmo) / 4); i += 32) d[i] = s[i];
    tm.sync();
}

// Gated: leaves if the block form took the launch (form_choice.cuh)
template <class TM, bool Gated>
__global__ void __launch_bounds__(256) fwd_structured_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo, DiscoebControl ctrl,
    int n_modes,
    const double* __restrict__ kmodes, const double* __restrict__ tau_start, const double* __restrict__ y0,
    const double* __restrict__ sw, int n_out, const double* __restrict__ tau_out, unsigned long long layout, int mem_doubles,
    int mix_doubles, double* y_full, double* y_out20, int32_t* status, int32_t* nsteps, int gate)
{
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5;
    const TM tm{(int)(threadIdx.x & 31)};
    if constexpr (Gated)
        if (short_chain_wins(tm, n_modes, kmodes, n_out, gate)) return;
    const int wpb = blockDim.x >> 5;
    double* base = smem + (size_t)warp * (kCosmoDoubles + mem_doubles + mix_doubles);
    DiscoebCosmo* P = reinterpret_cast<DiscoebCosmo*>(base);
    double* wmem = base + kCosmoDoubles;
    const int total_warps = gridDim.x * wpb;
    const int n0 = (mem_doubles - 4 * kMaxSlots - 32) / 23;  // state size of the launch (mode_mem_doubles)
    const double qnan = __longlong_as_double(0x7ff8000000000000LL);
    // outputs never reached are filled with NaN so that they cannot pass for data
    auto fill_nan = [&](int mode, int from) {
        for (int j = from; j < n_out; ++j) {
            const size_t o = (size_t)mode * n_out + j;
            if (y_full) for (int i = tm.lane; i < n0; i += 32) y_full[o * n0 + i] = qnan;
            if (y_out20) for (int i = tm.lane; i < 20; i += 32) y_out20[o * 20 + i] = qnan;
        }
    };
    int cur_cosmo = -1;
    for (int mode = blockIdx.x * wpb + warp; mode < n_modes; mode += total_warps) {
        const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
        if (bad_cosmology(cosmos, n_cosmo, ci, layout)) {  // invalid index or other sizes: report, solve nothing
            fill_nan(mode, 0);
            if (tm.leader()) {
                status[mode] = DISCOEB_BAD_INDEX;
                nsteps[mode] = 0;
            }
            continue;
        }
        if (ci != cur_cosmo) {
            copy_cosmo(tm, cosmos + ci, P);
            cur_cosmo = ci;
        }
        const Dims D = make_dims(*P);
        const int n = D.n;
        if (mode_mem_doubles(D) != mem_doubles || (TM::mixed && mixed_mem_doubles(D) != mix_doubles)) {
            // every cosmology must have the sizes of the first
            fill_nan(mode, 0);
            if (tm.leader()) {
                status[mode] = DISCOEB_BAD_INDEX;
                nsteps[mode] = 0;
            }
            continue;
        }
        ModeMem M = carve(wmem, D);
        if constexpr (TM::mixed) carve_mixed(wmem + mem_doubles, D, M);
        const double k = kmodes[mode];
        for (int i = tm.lane; i < n; i += 32) M.y[i] = y0[(size_t)mode * n + i];
        double swm[3] = {sw[3 * mode], sw[3 * mode + 1], sw[3 * mode + 2]};
        tm.sync();
        const size_t obase = (size_t)mode * n_out;
        const double* tout = tau_out + (size_t)ci * n_out;  // this cosmology's output times
        auto emit = [&](int j, const double* y, int) {
            const size_t o = obase + j;
            emit_output(tm, *P, D, k, tout[j], y, y_full ? y_full + o * n : nullptr,
                        y_out20 ? y_out20 + o * 20 : nullptr, M.f);
        };
        const SolveResult R = solve_mode(tm, *P, D, ctrl, k, tau_start[mode], swm, n_out, tout, M, emit);
        const int st = R.status, steps = R.steps;
        fill_nan(mode, R.outputs);
        if (tm.leader()) {
            status[mode] = st;
            nsteps[mode] = steps;
        }
        tm.sync();
    }
}

constexpr int kTanDoubles = (sizeof(DiscoebTangent) + 7) / 8;
constexpr int kMaxDirsPerBlock = 6;

// discoeb_jvp: one block per (mode, group of directions).  Warp 0 runs the adaptive forward
// solve and publishes every accepted step (start state, the 8 stages and the factorisation of
// W) into one of two shared-memory record slots; warps 1..nd each carry the tangent of one
// direction through the published steps (tangent_step) and write its outputs.  The forward
// is solved once per block instead of once per direction, and it runs ahead of the tangents
// by up to two steps.  Steps are handed over with counters in shared memory (published /
// consumed), every wait bounded (wait_at_least); if a wait gives up, the whole block stops and
// reports DISCOEB_ABORTED.  The step sequence is the forward's only, so the tangent is the
// derivative of the discrete solution with the accepted steps held fixed.
//
// Split and shared records give the same bits (a test compares them), which hangs on the compiler fusing the
// same multiply-adds in both: one number for the layout instead of the sizes, or the gate's test in every
// instantiation, turns a choice over in one of them (2e-13).
template <bool Full, bool Split, bool Gated>
__global__ void __launch_bounds__(32 * (1 + kMaxDirsPerBlock)) jvp_block_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo,
    const DiscoebTangent* __restrict__ tangents, int n_dir, int dpb, Dims D0,
    DiscoebControl ctrl, int n_modes, const double* __restrict__ kmodes, const double* __restrict__ tau_start,
    const double* __restrict__ y0, const double* __restrict__ y0_dot, const double* __restrict__ sw, int n_out,
    const double* __restrict__ tau_out, const double* __restrict__ tau_out_dot, int mem_doubles, int tan_doubles,
    double* rec_glob, double* y_out20, double* y_out20_dot, int32_t* status, int32_t* nsteps, int gate)
{
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5;
    WarpTeamSeq tm;
    tm.lane = (int)(threadIdx.x & 31);
    if constexpr (Gated)
        if (short_chain_wins(tm, n_modes, kmodes, n_out, gate)) return;
    const int groups = (n_dir + dpb - 1) / dpb;
    const int mode = blockIdx.x / groups, grp = blockIdx.x - mode * groups;
    const int d0 = grp * dpb, nd = min(dpb, n_dir - d0);
    const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
    if (ci < 0 || ci >= n_cosmo) {  // invalid cosmology index: report, solve nothing
        const double qn = __longlong_as_double(0x7ff8000000000000LL);
        if (threadIdx.x == 0 && grp == 0) {
            status[mode] = DISCOEB_BAD_INDEX;
            nsteps[mode] = 0;
        }
        // outputs of width 20 (fields) or, for Full, the state size of the first cosmology
        const int W = Full ? D0.n : 20;
        for (int dd = 0; dd < nd; ++dd)
            for (int i = threadIdx.x; i < n_out * W; i += blockDim.x) {
                y_out20_dot[((size_t)(d0 + dd) * n_modes + mode) * n_out * W + i] = qn;
                if (d0 + dd == 0 && y_out20) y_out20[(size_t)mode * n_out * W + i] = qn;
            }
        return;
    }
    const DiscoebCosmo* cosmo = cosmos + ci;
    tangents += (size_t)ci * n_dir;
    tau_out += (size_t)ci * n_out;
    tau_out_dot += (size_t)ci * n_dir * n_out;
    // shared layout: cosmology, tangents, forward workspace, two step records (+4 scalars
    // each: t, h, t_next, regime), per tangent warp its workspace + 3 n doubles, flags.  With
    // rec_glob (for states whose records would leave room for fewer tangent warps) there is one
    // record, split: its first 13 n doubles (state, stage vectors) in the block's own part of that
    // global array, the factorisation of W (10 n + 224 doubles, re-read by every stage's solve)
    // and the scalars in shared memory; the forward runs one step ahead instead of two
    DiscoebCosmo* P = reinterpret_cast<DiscoebCosmo*>(smem);
    DiscoebTangent* TNs = reinterpret_cast<DiscoebTangent*>(smem + kCosmoDoubles);
    double* fmem = smem + kCosmoDoubles + dpb * kTanDoubles;
    const int rec = mem_doubles + 4;
    const int n0 = D0.n;  // state size
    constexpr int ns = Split ? 1 : 2;            // record slots
    const int gpart = Split ? 13 * n0 : 0;       // doubles of a record in global memory
    const int spart = rec - gpart;               // doubles of a record in shared memory
    double* gslot = Split ? rec_glob + (size_t)blockIdx.x * gpart : nullptr;
    double* slot0 = fmem + mem_doubles;
    const int per_tan = tan_doubles + 3 * n0;
    double* twork = slot0 + ns * spart;
    int* flags = reinterpret_cast<int*>(twork + (size_t)dpb * per_tan);
    // flags: [0,1] published count per slot (step m + 1), [2,3] consumptions per slot,
    //        [4] forward finished, [5] published steps in total, [6] abort
    volatile int* vf = flags;
    {
        const int* s = reinterpret_cast<const int*>(cosmo);
        int* d = reinterpret_cast<int*>(P);
        for (int i = threadIdx.x; i < (int)(sizeof(DiscoebCosmo) / 4); i += blockDim.x) d[i] = s[i];
        for (int dd = 0; dd < nd; ++dd) {
            const int* ts = reinterpret_cast<const int*>(tangents + d0 + dd);
            int* td = reinterpret_cast<int*>(TNs + dd);
            for (int i = threadIdx.x; i < (int)(sizeof(DiscoebTangent) / 4); i += blockDim.x) td[i] = ts[i];
        }
        if (threadIdx.x < 8) flags[threadIdx.x] = 0;
    }
    __syncthreads();
    if (warp > nd) return;  // surplus warps of the last group
    const Dims D = make_dims(*P);
    const int n = D.n;
    if (!same_layout(D, D0)) {  // every cosmology must have the sizes of the first
        const double qn = __longlong_as_double(0x7ff8000000000000LL);
        if (warp == 0) {
            if (tm.leader() && grp == 0) {
                status[mode] = DISCOEB_BAD_INDEX;
                nsteps[mode] = 0;
            }
        } else {
            const int dir = d0 + warp - 1;
            const int W = Full ? D0.n : 20;
            for (int i = tm.lane; i < n_out * W; i += 32) {
                y_out20_dot[((size_t)dir * n_modes + mode) * n_out * W + i] = qn;
                if (dir == 0 && y_out20) y_out20[(size_t)mode * n_out * W + i] = qn;
            }
        }
        return;
    }
    const double k = kmodes[mode];
    const double* tout = tau_out;
    const double qnan = __longlong_as_double(0x7ff8000000000000LL);

    if (warp == 0) {
        // ---- forward: solve, publish every accepted step ----
        ModeMem M = carve(fmem, D);
        for (int i = tm.lane; i < n; i += 32) M.y[i] = y0[(size_t)mode * n + i];
        double swm[3] = {sw[3 * mode], sw[3 * mode + 1], sw[3 * mode + 2]};
        tm.sync();
        int m = 0;
        auto accept = [&](double t, double h, double tnext, int regime) -> bool {
            const int sl = m % ns;
            if (m >= ns && !wait_at_least(tm, vf + 2 + sl, nd * (m / ns), vf + 6, poll_budget(ctrl))) return false;
            double* dst = slot0 + sl * spart;
            if (Split)
                for (int i = tm.lane; i < gpart; i += 32) gslot[i] = fmem[i];
            for (int i = tm.lane; i < mem_doubles - gpart; i += 32) dst[i] = fmem[gpart + i];
            if (tm.leader()) {
                dst[spart - 4] = t;
                dst[spart - 3] = h;
                dst[spart - 2] = tnext;
                dst[spart - 1] = (double)regime;
            }
            tm.sync();
            if (tm.leader()) {
                __threadfence_block();
                vf[sl] = m + 1;
            }
            tm.sync();
            ++m;
            return true;
        };
        auto no_emit = [&](int, const double*, int) {};
        const SolveResult R = solve_mode(tm, *P, D, ctrl, k, tau_start[mode], swm, n_out, tout, M, no_emit,
                                         (const DiscoebTangent*)nullptr, (const TanMem*)nullptr, (double*)nullptr, 0,
                                         &accept);
        if (tm.leader()) {
            vf[5] = m;
            __threadfence_block();
            vf[4] = 1;
            if (grp == 0) nsteps[mode] = R.steps;
        }
        tm.sync();
        report_status(tm, R.status, m, ns, nd, vf + 2, vf + 6, poll_budget(ctrl), groups > 1, status + mode);
        return;
    }

    // ---- tangent of direction d0 + warp - 1 ----
    const int dl = warp - 1, dir = d0 + dl;
    const DiscoebTangent* TN = TNs + dl;
    double* mine = twork + (size_t)dl * per_tan;
    const TanMem TT = carve_tan(mine, D);
    double* ubuf = mine + tan_doubles;
    double* yend = ubuf + n;
    double* pf = yend + n;
    for (int i = tm.lane; i < n; i += 32) TT.yd[i] = y0_dot[((size_t)dir * n_modes + mode) * n + i];
    tm.sync();
    int hint = P->xe_loga.n_knots / 2, iout = 0;
    const long long budget = poll_budget(ctrl);
    for (int m = 0;; ++m) {
        const int sl = m % ns;
        // the next step, unless the forward has finished with fewer steps
        int have = 0;
        if (tm.leader()) {
            long long polls = 0;
            while (true) {
                if (vf[sl] == m + 1) { have = 1; break; }
                if (vf[4] && vf[5] <= m) break;
                if (vf[6]) break;
                if (++polls > budget) { vf[6] = 1; break; }
                __nanosleep(100);
            }
            __threadfence_block();
        }
        if (!__shfl_sync(0xffffffffu, have, 0)) break;
        const double* r = slot0 + sl * spart;
        ModeMem Mr = Split ? carve_split(gslot, const_cast<double*>(r), D) : carve(const_cast<double*>(r), D);
        Mr.u = ubuf;
        const double t = r[spart - 4], h = r[spart - 3], tnext = r[spart - 2];
        const int regime = (int)r[spart - 1];
        tangent_step(tm, *P, D, k, t, h, regime, Mr, TT, TN, hint);
        for (int i = tm.lane; i < n; i += 32) yend[i] = ubuf[i] + Mr.K[7 * n + i];
        tm.sync();
        if (tm.leader()) {
            __threadfence_block();
            atomicAdd(flags + 2 + sl, 1);  // the record may be overwritten from here on
        }
        tm.sync();
        while (iout < n_out && tout[iout] <= tnext) {
            emit_tangent_output<Full>(tm, *P, TN, D, k, mode, dir, n_modes, n_out, iout, tout, tau_out_dot, yend,
                                      regime, TT, pf, y_out20, y_out20_dot);
            ++iout;
        }
    }
    constexpr int W20 = 20;
    const int W = Full ? n : W20;
    for (int j = iout; j < n_out; ++j) {
        const size_t oo = (size_t)mode * n_out + j;
        for (int i = tm.lane; i < W; i += 32) {
            y_out20_dot[((size_t)dir * n_modes * n_out + oo) * W + i] = qnan;
            if (dir == 0 && y_out20) y_out20[oo * W + i] = qnan;
        }
    }
    tm.sync();
}

__global__ void rhs_kernel(const DiscoebCosmo* __restrict__ cosmo, int n_points, const double* __restrict__ tau,
                           const double* __restrict__ kmodes, const double* __restrict__ y, int regime, double* f)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= n_points) return;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const DiscoebCosmo& P = *cosmo;
    const Dims D = make_dims(P);
    const double* yy = y + (size_t)warp * D.n;
    Bg<double> b;
    bg_eval(P, yy[0], tau[warp], kmodes[warp], regime, b);
    rhs_team(tm, P, D, b, kmodes[warp], tau[warp], yy, f + (size_t)warp * D.n, (double*)nullptr);
}

int validate_cosmo(const DiscoebCosmo* c)
{
    if (!c) return DISCOEB_EINVAL;
    if (c->nqmax < 0 || c->nqmax > DISCOEB_MAX_NQ) return DISCOEB_EINVAL;
    if (c->lmaxg < 3 || c->lmaxgp < 3 || c->lmaxr < 3 || c->lmaxnu < 3) return DISCOEB_EINVAL;
    if (c->use_tca) return DISCOEB_EUNSUPPORTED;
    return DISCOEB_SUCCESS;
}

// Directions per block of discoeb_jvp: as many as fit in shared memory (at most
// kMaxDirsPerBlock; the forward is solved once per block).  With the two step records in shared
// memory (dpb, smem), or in a global workspace (dpb_glob, smem_glob), which is worth its
// records_bytes only when it lets more directions share a block (larger states, e.g. l_max 50).
struct JvpPlan {
    int dpb, dpb_glob, mem, tmem;
    size_t smem, smem_glob;
    int64_t records_bytes;  // recommended: the split form's workspace where it adds directions, else 0
    int64_t split_bytes;    // the split form's workspace (a caller may ask for it anyway)
};

JvpPlan jvp_plan(const DiscoebCosmo& c0, int n_dir, int n_modes)
{
    JvpPlan p{};
    const Dims D = make_dims(c0);
    p.mem = mode_mem_doubles(D);
    p.tmem = tan_mem_doubles(D);
    int dev = 0, max_optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        p.dpb = -1;
        return p;
    }
    // shared doubles: cosmology, tangents, forward workspace, the records' shared parts (two
    // whole records, or one record's factorisation and scalars), the tangent warps' workspaces
    auto bytes = [&](int d, bool glob) {
        const size_t recs = glob ? (size_t)(p.mem + 4 - 13 * D.n) : 2 * (size_t)(p.mem + 4);
        return (size_t)(kCosmoDoubles + d * kTanDoubles + p.mem + recs + d * (p.tmem + 3 * D.n)) * sizeof(double) +
               8 * sizeof(int);
    };
    const int want = n_dir < kMaxDirsPerBlock ? n_dir : kMaxDirsPerBlock;
    auto fit = [&](bool glob) {
        int d = want;
        while (d > 1 && bytes(d, glob) > (size_t)max_optin) --d;
        return bytes(d, glob) <= (size_t)max_optin ? d : 0;
    };
    p.dpb = fit(false);
    p.dpb_glob = fit(true);
    p.smem = bytes(p.dpb > 0 ? p.dpb : 1, false);
    p.smem_glob = bytes(p.dpb_glob > 0 ? p.dpb_glob : 1, true);
    if (p.dpb_glob > 0) {
        const long long blocks = (long long)n_modes * ((n_dir + p.dpb_glob - 1) / p.dpb_glob);
        p.split_bytes = blocks * 13LL * D.n * (int64_t)sizeof(double);
    }
    if (p.dpb_glob > p.dpb) p.records_bytes = p.split_bytes;
    return p;
}

// The block of warps (nd directions a block) against jvp_block_kernel (dpb).  Its chain is a third as
// long, but where shared memory holds few directions beside it the forward runs once more per group of
// them.  Milliseconds, block / older, k from 1e-4 to 1, six directions, 1000 modes: twice the groups still
// win (93 to 156 rows 275 / 370, 144 rows 262 / 364, 194 rows 290 / 834); three times and more do not
// (161 rows 475 / 384, 121 rows of 8 bins 835 / 377, 219 rows 903 / 842), where few modes do (161 rows, 80
// modes 37.5 / 82.2; equal k, 49 modes 90 / 192, 148 modes 286 / 205).
// - Against the split record at one direction a block (219 rows, whole states): 600 modes to k = 0.5, 40
//   outputs 576 / 664 (to k = 1), 320 outputs 1027 / 930, 2000 outputs 4409 / 3529, but 300 modes 505 / 522 and 80
//   modes 703 / 803: each of the six forwards stops at every output.
// - Many whole states favour the block, which projects them afterwards: 161 rows, 320 outputs 501 / 545.
// - One direction asked for: the older form then has several blocks per SM (72 rows, 1000 modes 164 / 124;
//   99 rows 173 / 179, 143 rows 164 / 213).
FormChoice jvp_choice(const Dims& D, int n_dir, int nd, int dpb, bool split, bool full, int n_out, int n_modes, int sms)
{
    const int groups = (n_dir + nd - 1) / nd, older = dpb > 0 ? (n_dir + dpb - 1) / dpb : 0;
    long long limit = n_modes;  // (the block form only)
    if (dpb == 0) return FormChoice(n_modes, limit);
    if (split) {
        if (groups > 1 && nd == 1 && n_out > 128) limit = 3LL * sms / 2;
    } else if (n_dir == 1 && D.n < 99) {
        limit = sms;
    } else if (groups > (full && n_out > 128 ? 3 : 2) * older) {
        limit = 2LL * sms * older / groups;
    }
    return FormChoice(n_modes, limit);
}

template <bool Full>
int32_t launch_jvp(const DiscoebCosmo* cosmos_dev, const DiscoebCosmo* cosmo0_host, int32_t n_cosmo,
                   const int32_t* mode_cosmo, const DiscoebTangent* tangents_dev, int32_t n_dir,
                   const DiscoebControl* ctrl, int32_t n_modes, const double* kmodes, const double* tau_start,
                   const double* y0, const double* y0_dot, const double* switch_tau, int32_t n_out,
                   const double* tau_out, const double* tau_out_dot, double* y_out, double* y_out_dot,
                   int32_t* status, int32_t* nsteps, double* records, int64_t records_bytes, void* stream)
{
    int rc = validate_cosmo(cosmo0_host);
    if (rc) return rc;
    if (!cosmos_dev || !ctrl || !tangents_dev || n_cosmo < 1 || n_dir < 1 || n_modes < 0 || n_out < 1)
        return DISCOEB_EINVAL;
    if (n_modes == 0) return DISCOEB_SUCCESS;
    if (!kmodes || !tau_start || !y0 || !y0_dot || !switch_tau || !tau_out || !tau_out_dot || !y_out_dot ||
        !status || !nsteps)
        return DISCOEB_EINVAL;
    if (ctrl->method != DISCOEB_METHOD_RODAS5_STRUCTURED) return DISCOEB_EUNSUPPORTED;
    if (!(ctrl->rtol > 0.0) || !(ctrl->atol >= 0.0) || ctrl->max_steps < 1) return DISCOEB_EINVAL;
    int dev = 0, max_optin = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // the split record is used when the caller passes room for it (discoeb_jvp_records_bytes
    // recommends it where it lets more directions share a block; a caller may pass it anyway)
    const JvpPlan plan = jvp_plan(*cosmo0_host, n_dir, n_modes);
    if (plan.dpb < 0) return DISCOEB_ECUDA;
    const bool glob = plan.dpb_glob >= plan.dpb && plan.split_bytes > 0 && records && records_bytes >= plan.split_bytes;
    int gate = FormChoice::kOnly;
    size_t bsmem = 0;
    const Dims D = make_dims(*cosmo0_host);
    const int bnd = blk::jvp_directions(D, n_dir < kMaxDirsPerBlock ? n_dir : kMaxDirsPerBlock, (size_t)max_optin, bsmem);
    if (bnd > 0) {
        const FormChoice form = jvp_choice(D, n_dir, bnd, glob ? plan.dpb_glob : plan.dpb, glob, Full, n_out, n_modes, sms);
        gate = form.gate();
        if (form.short_chain) {
            rc = blk::launch_jvp_block<Full>(cosmos_dev, n_cosmo, mode_cosmo, tangents_dev, n_dir, bnd, bsmem, D, *ctrl,
                                             n_modes, kmodes, tau_start, y0, y0_dot, switch_tau, n_out, tau_out,
                                             tau_out_dot, y_out, y_out_dot, status, nsteps, gate,
                                             reinterpret_cast<cudaStream_t>(stream));
            if (rc || !form.many_modes) return rc;
        }
    }
    if (!glob && plan.dpb == 0) return DISCOEB_EUNSUPPORTED;
    const int dpb = glob ? plan.dpb_glob : plan.dpb;
    const size_t smem = glob ? plan.smem_glob : plan.smem;
    const int mem = plan.mem, tmem = plan.tmem;
    const auto pick = [&](auto shared, auto split) { return glob ? split : shared; };
    const auto kernel = gate == FormChoice::kOnly
                            ? pick(jvp_block_kernel<Full, false, false>, jvp_block_kernel<Full, true, false>)
                            : pick(jvp_block_kernel<Full, false, true>, jvp_block_kernel<Full, true, true>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DISCOEB_ECUDA;
    const long long blocks = (long long)n_modes * ((n_dir + dpb - 1) / dpb);
    if (blocks > 0x7fffffffLL) return DISCOEB_EINVAL;
    // (several blocks report a mode: report_status; after the block form's kernel it holds kOtherForm)
    if (blocks > n_modes && gate == FormChoice::kOnly &&
        cudaMemsetAsync(status, 0, (size_t)n_modes * sizeof(int32_t), reinterpret_cast<cudaStream_t>(stream)) !=
            cudaSuccess)
        return DISCOEB_ECUDA;
    kernel<<<(unsigned)blocks, 32 * (1 + dpb), smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        cosmos_dev, n_cosmo, mode_cosmo, tangents_dev, n_dir, dpb, D, *ctrl, n_modes, kmodes, tau_start, y0,
        y0_dot, switch_tau, n_out, tau_out, tau_out_dot, mem, tmem, glob ? records : nullptr, y_out, y_out_dot, status,
        nsteps, gate);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

}  // namespace

extern "C" {

int32_t discoeb_abi_version(void) { return DISCOEB_ABI_VERSION; }

int32_t discoeb_nvar(const DiscoebCosmo* cosmo)
{
    if (!cosmo) return DISCOEB_EINVAL;
    return make_dims(*cosmo).n;
}

int32_t discoeb_fwd(const DiscoebCosmo* cosmos_dev, const DiscoebCosmo* cosmo0_host, int32_t n_cosmo,
                    const DiscoebControl* ctrl, int32_t n_modes, const int32_t* mode_cosmo, const double* kmodes,
                    const double* tau_start, const double* y0, const double* switch_tau, int32_t n_out,
                    const double* tau_out, double* y_full, double* y_out20, int32_t* status, int32_t* nsteps,
                    void* stream)
{
    int rc = validate_cosmo(cosmo0_host);
    if (rc) return rc;
    if (!cosmos_dev || !ctrl || n_cosmo < 1 || n_modes < 0 || n_out < 1) return DISCOEB_EINVAL;
    if (n_modes == 0) return DISCOEB_SUCCESS;
    if (!kmodes || !tau_start || !y0 || !switch_tau || !tau_out || !status || !nsteps) return DISCOEB_EINVAL;
    if (!y_full && !y_out20) return DISCOEB_EINVAL;
    const bool mixed = ctrl->method == DISCOEB_METHOD_RODAS5_STRUCTURED_MIXED;
    if (ctrl->method != DISCOEB_METHOD_RODAS5_STRUCTURED && !mixed) return DISCOEB_EUNSUPPORTED;
    if (!(ctrl->rtol > 0.0) || !(ctrl->atol >= 0.0) || ctrl->max_steps < 1) return DISCOEB_EINVAL;
    const Dims D = make_dims(*cosmo0_host);
    const int mem = mode_mem_doubles(D), mix = mixed ? mixed_mem_doubles(D) : 0;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    int max_optin = 0;
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // FP64: a block of warps per mode, up to the work where one warp per mode has more of them in flight;
    // the same results bit for bit
    int gate = FormChoice::kOnly;
    if (!mixed && blk::smem_bytes(D) <= (size_t)max_optin) {
        const FormChoice form = blk::forward_choice(D, n_modes, sms);
        gate = form.gate();
        if (form.short_chain) {
            rc = blk::launch_fwd(cosmos_dev, n_cosmo, mode_cosmo, *ctrl, n_modes, kmodes, tau_start, y0, switch_tau,
                                 n_out, tau_out, D, y_full, y_out20, status, nsteps, nullptr, sms, gate, s);
            if (rc || !form.many_modes) return rc;
        }
    }
    const size_t per_warp = (size_t)(kCosmoDoubles + mem + mix) * sizeof(double);
    const auto kernel = mixed                        ? fwd_structured_kernel<WarpTeamMixed, false>
                        : gate != FormChoice::kOnly ? fwd_structured_kernel<WarpTeam, true>
                                                    : fwd_structured_kernel<WarpTeam, false>;
    int wpb = ctrl->warps_per_block > 0 ? ctrl->warps_per_block : 1;  // one mode per block: the most resident warps
    if (wpb > 8) wpb = 8;
    while (wpb > 1 && per_warp * wpb > (size_t)max_optin) --wpb;
    if (per_warp > (size_t)max_optin) return DISCOEB_EUNSUPPORTED;
    const size_t smem = per_warp * wpb;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DISCOEB_ECUDA;
    int blocks = (n_modes + wpb - 1) / wpb;
    kernel<<<blocks, 32 * wpb, smem, s>>>(cosmos_dev, n_cosmo, mode_cosmo, *ctrl, n_modes, kmodes, tau_start, y0,
                                          switch_tau, n_out, tau_out, layout_key(D), mem, mix, y_full, y_out20, status,
                                          nsteps, gate);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int32_t discoeb_jvp(const DiscoebCosmo* cosmos_dev, const DiscoebCosmo* cosmo0_host, int32_t n_cosmo,
                    const int32_t* mode_cosmo, const DiscoebTangent* tangents_dev,
                    int32_t n_dir, const DiscoebControl* ctrl, int32_t n_modes, const double* kmodes,
                    const double* tau_start, const double* y0, const double* y0_dot, const double* switch_tau,
                    int32_t n_out, const double* tau_out, const double* tau_out_dot, double* y_out20,
                    double* y_out20_dot, int32_t* status, int32_t* nsteps, void* stream)
{
    return launch_jvp<false>(cosmos_dev, cosmo0_host, n_cosmo, mode_cosmo, tangents_dev, n_dir, ctrl, n_modes, kmodes,
                             tau_start, y0, y0_dot, switch_tau, n_out, tau_out, tau_out_dot, y_out20, y_out20_dot,
                             status, nsteps, nullptr, 0, stream);
}

int32_t discoeb_jvp_full(const DiscoebCosmo* cosmos_dev, const DiscoebCosmo* cosmo0_host, int32_t n_cosmo,
                         const int32_t* mode_cosmo, const DiscoebTangent* tangents_dev, int32_t n_dir,
                         const DiscoebControl* ctrl, int32_t n_modes, const double* kmodes, const double* tau_start,
                         const double* y0, const double* y0_dot, const double* switch_tau, int32_t n_out,
                         const double* tau_out, const double* tau_out_dot, double* y_full, double* y_full_dot,
                         int32_t* status, int32_t* nsteps, void* stream)
{
    return launch_jvp<true>(cosmos_dev, cosmo0_host, n_cosmo, mode_cosmo, tangents_dev, n_dir, ctrl, n_modes, kmodes,
                            tau_start, y0, y0_dot, switch_tau, n_out, tau_out, tau_out_dot, y_full, y_full_dot,
                            status, nsteps, nullptr, 0, stream);
}

int64_t discoeb_jvp_records_bytes(const DiscoebCosmo* cosmo0_host, int32_t n_dir, int32_t n_modes)
{
    if (validate_cosmo(cosmo0_host) || n_dir < 1 || n_modes < 0) return DISCOEB_EINVAL;
    const JvpPlan plan = jvp_plan(*cosmo0_host, n_dir, n_modes);
    return plan.dpb < 0 ? (int64_t)DISCOEB_ECUDA : plan.records_bytes;
}

int64_t discoeb_jvp_split_records_bytes(const DiscoebCosmo* cosmo0_host, int32_t n_dir, int32_t n_modes)
{
    if (validate_cosmo(cosmo0_host) || n_dir < 1 || n_modes < 0) return DISCOEB_EINVAL;
    const JvpPlan plan = jvp_plan(*cosmo0_host, n_dir, n_modes);
    return plan.dpb < 0 ? (int64_t)DISCOEB_ECUDA : plan.split_bytes;
}

int32_t discoeb_jvp_records(const DiscoebCosmo* cosmos_dev, const DiscoebCosmo* cosmo0_host, int32_t n_cosmo,
                            const int32_t* mode_cosmo, const DiscoebTangent* tangents_dev, int32_t n_dir,
                            const DiscoebControl* ctrl, int32_t n_modes, const double* kmodes, const double* tau_start,
                            const double* y0, const double* y0_dot, const double* switch_tau, int32_t n_out,
                            const double* tau_out, const double* tau_out_dot, double* y_out, double* y_out_dot,
                            int32_t* status, int32_t* nsteps, int32_t full, void* records, int64_t records_bytes,
                            void* stream)
{
    if (full != 0 && full != 1) return DISCOEB_EINVAL;
    double* rec = static_cast<double*>(records);
    if (full)
        return launch_jvp<true>(cosmos_dev, cosmo0_host, n_cosmo, mode_cosmo, tangents_dev, n_dir, ctrl, n_modes,
                                kmodes, tau_start, y0, y0_dot, switch_tau, n_out, tau_out, tau_out_dot, y_out,
                                y_out_dot, status, nsteps, rec, records_bytes, stream);
    return launch_jvp<false>(cosmos_dev, cosmo0_host, n_cosmo, mode_cosmo, tangents_dev, n_dir, ctrl, n_modes, kmodes,
                             tau_start, y0, y0_dot, switch_tau, n_out, tau_out, tau_out_dot, y_out, y_out_dot, status,
                             nsteps, rec, records_bytes, stream);
}

int32_t discoeb_rhs(const DiscoebCosmo* cosmo_dev, const DiscoebCosmo* cosmo_host, int32_t n_points,
                    const double* tau, const double* kmodes, const double* y, int32_t regime, double* f, void* stream)
{
    int rc = validate_cosmo(cosmo_host);
    if (rc) return rc;
    if (!cosmo_dev || n_points < 0) return DISCOEB_EINVAL;
    if (n_points == 0) return DISCOEB_SUCCESS;
    if (!tau || !kmodes || !y || !f) return DISCOEB_EINVAL;
    const int threads = 128;
    const long long blocks = ((long long)n_points * 32 + threads - 1) / threads;
    rhs_kernel<<<(unsigned)blocks, threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(cosmo_dev, n_points, tau,
                                                                                          kmodes, y, regime, f);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

}  // extern "C"
