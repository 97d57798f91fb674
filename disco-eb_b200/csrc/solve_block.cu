// Forward perturbation solve, FP64, a block of warps per mode: kernels and launch of discoeb_fwd.
#define DSCB_CALL_MATH
#include <cuda_runtime.h>

#include "discoeb.h"
#include "emit_output.cuh"
#include "solve_block.cuh"
#include "solve_block_launch.cuh"

using namespace dscb;

namespace {

// discoeb_fwd, FP64 form: a block of cooperating warps per mode (solve_block.cuh).  With whole states
// asked for, the solve stores them as they are and project_states_kernel applies the RSA
// projection afterwards, one warp per (mode, output): 320 projections per mode would otherwise sit
// on the mode's chain of steps.
//
// Record: the recording forward of the adjoint.  Each accepted step's end time and every `every`-th
// start state go into the mode's record (record_doubles), by the controller's warp before the state
// advances.
template <int MaxThreads, int MinBlocks, bool Record>
__global__ void __launch_bounds__(MaxThreads, MinBlocks) fwd_block_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo, DiscoebControl ctrl,
    const double* __restrict__ kmodes, const double* __restrict__ tau_start, const double* __restrict__ y0,
    const double* __restrict__ sw, int n_out, const double* __restrict__ tau_out, Dims D0, double* y_full,
    double* y_out20, int32_t* status, int32_t* nsteps, blk::StepRecords rec, int gate)
{
    extern __shared__ double smem[];
    DiscoebCosmo* P = reinterpret_cast<DiscoebCosmo*>(smem);
    blk::Shared& S = *reinterpret_cast<blk::Shared*>(smem + blk::kCosmo);
    double* wmem = smem + blk::kCosmo + blk::kSharedDoubles;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int mode = blockIdx.x, warp = threadIdx.x >> 5;
    if (gate != FormChoice::kOnly && !short_chain_wins(tm, gridDim.x, kmodes, n_out, gate)) {
        if (threadIdx.x == 0) status[mode] = kOtherForm;
        return;
    }
    const double qnan = __longlong_as_double(0x7ff8000000000000LL);
    // outputs never reached are filled with NaN so that they cannot pass for data
    auto fill_nan = [&](int from) {
        for (int j = from; j < n_out; ++j) {
            const size_t o = (size_t)mode * n_out + j;
            if (y_full) for (int i = tm.lane; i < D0.n; i += 32) y_full[o * D0.n + i] = qnan;
            if (y_out20) for (int i = tm.lane; i < 20; i += 32) y_out20[o * 20 + i] = qnan;
        }
    };
    const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
    bool bad = ci < 0 || ci >= n_cosmo;  // invalid cosmology index: report, solve nothing
    if (!bad) {
        const int* src = reinterpret_cast<const int*>(cosmos + ci);
        int* dst = reinterpret_cast<int*>(P);
        for (int i = threadIdx.x; i < (int)(sizeof(DiscoebCosmo) / 4); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    Dims D{};
    if (!bad) {
        D = make_dims(*P);
        bad = !same_layout(D, D0);  // every cosmology must have the sizes of the first
    }
    if (bad) {
        if (warp == 0) fill_nan(0);
        if (threadIdx.x == 0) {
            status[mode] = DISCOEB_BAD_INDEX;
            nsteps[mode] = 0;
            if constexpr (Record) rec.n_accepted[mode] = 0;
        }
        return;
    }
    const int n = D.n;
    const ModeMem M = blk::block_carve(wmem, D);
    const double k = kmodes[mode];
    for (int i = threadIdx.x; i < n; i += blockDim.x) M.y[i] = y0[(size_t)mode * n + i];
    const double swm[3] = {sw[3 * mode], sw[3 * mode + 1], sw[3 * mode + 2]};
    const double* tout = tau_out + (size_t)ci * n_out;  // this cosmology's output times
    __syncthreads();
    auto emit = [&](int j, const double* y) {
        if (!y_full && (!Record || y_out20))
            emit_output(tm, *P, D, k, tout[j], y, nullptr, y_out20 + ((size_t)mode * n_out + j) * 20, M.f);
    };
    auto rows = [&](int j, int i, double v) {
        if (y_full) y_full[((size_t)mode * n_out + j) * n + i] = v;
    };
    int count = 0;
    auto accept = [&](double, double, double tnext, int) {
        if constexpr (Record) {
            if (count >= rec.cap) return false;
            double* r = rec.base + (size_t)mode * rec.doubles;
            if (count % rec.every == 0) {
                double* c = r + rec.cap + (size_t)(count / rec.every) * n;
                for (int i = tm.lane; i < n; i += 32) c[i] = M.y[i];
            }
            if (tm.leader()) r[count] = tnext;
            ++count;
        }
        return true;
    };
    const SolveResult R = blk::solve_mode_block(*P, D, ctrl, k, tau_start[mode], swm, n_out, tout, M, S, emit, rows,
                                                accept);
    if (warp == 0) {
        fill_nan(R.outputs);
        if (tm.leader()) {
            status[mode] = (Record && R.status == DISCOEB_ABORTED && count >= rec.cap) ? DISCOEB_RECORD_FULL : R.status;
            nsteps[mode] = R.steps;
            if constexpr (Record) rec.n_accepted[mode] = count;
        }
    }
}

// The RSA projection of the states fwd_block_kernel stored (in place), and their output fields when
// asked for: one warp per (mode, output); rows never reached hold NaN and stay as they are.
__global__ void __launch_bounds__(128) project_states_kernel(
    const DiscoebCosmo* __restrict__ cosmos, int n_cosmo, const int32_t* __restrict__ mode_cosmo, long long n_points,
    const double* __restrict__ kmodes, int n_out, const double* __restrict__ tau_out, Dims D0, const int32_t* __restrict__ status,
    double* y_full, double* y_out20)
{
    const long long p = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= n_points) return;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int mode = (int)(p / n_out), j = (int)(p - (long long)mode * n_out);
    const int ci = mode_cosmo ? mode_cosmo[mode] : 0;
    if (ci < 0 || ci >= n_cosmo) return;
    const DiscoebCosmo& P = cosmos[ci];
    const Dims D = make_dims(P);
    if (!same_layout(D, D0) || status[mode] == kOtherForm) return;
    const int n0 = D0.n;
    double* y = y_full + (size_t)p * n0;
    if (!(y[0] == y[0])) return;
    const double k = kmodes[mode], tau = tau_out[(size_t)ci * n_out + j];
    double fld[4];
    const bool rsa = rsa_projection<double>(P, nullptr, D, tau, k, y, nullptr, fld);  // all lanes, identical
    tm.sync();
    if (rsa)
        for (int i = tm.lane; i < n0; i += 32) {
            const int s = rsa_slot(D, i);
            if (s >= 0) y[i] = fld[s];
            else if (s == -1) y[i] = 0.0;
        }
    tm.sync();
    if (y_out20 && tm.leader()) {
        double o[20];
        output_vars<double>(P, nullptr, D, k, y, nullptr, o);
        for (int q = 0; q < 20; ++q) y_out20[(size_t)p * 20 + q] = o[q];
    }
}

}  // namespace

namespace dscb {
namespace blk {

size_t smem_bytes(const Dims& D)
{
    return block_threads(D) > 512 ? ~(size_t)0 : (size_t)smem_doubles(D) * sizeof(double);
}

// Modes of equal length per SM up to which blocks (two at a time) beat a warp per mode (8 to 16 of them),
// from the equal times: 2.8 for 25 rows, 4.2 for 72, 5.2 for 143; with more than five momentum bins, whose
// chains are wider, 2.7 to 4.0 for 85 to 197 rows; above 256 threads, one block per SM, 3.7 to 4.0 for 144
// to 219 rows.  Milliseconds, block / one-warp: k from 1e-4 to 5, 72 rows, 1024 modes 43 / 98; 143 rows, 2048
// modes 79 / 111, with 15 bins 3072 modes 186 / 118; 144 rows, 1024 modes 65 / 112, 2048 modes 128 / 115, 4096
// modes 259 / 151; equal k, 1024 modes of 72 rows 167 / 105, of 143 rows 145 / 114, of 144 rows 212 / 120.
// Up to 3.5 modes per SM a block has the SM to itself and modes of equal length finish in whole rounds.
FormChoice forward_choice(const Dims& D, int n_modes, int sms)
{
    int tenths = 23 + D.n / 5;
    if (chain_stride(D) != kNarrow) tenths = tenths < 29 ? tenths : 29;
    else if (block_threads(D) > 256) tenths = 37;
    if (2LL * n_modes <= 7LL * sms) tenths -= tenths % 10;
    return FormChoice(n_modes, (long long)tenths * sms / 10);
}

int32_t launch_fwd(const DiscoebCosmo* cosmos, int n_cosmo, const int32_t* mode_cosmo, const DiscoebControl& ctrl,
                   int n_modes, const double* kmodes, const double* tau_start, const double* y0, const double* sw,
                   int n_out, const double* tau_out, const Dims& D, double* y_full, double* y_out20, int32_t* status,
                   int32_t* nsteps, const StepRecords* records, int sms, int gate, cudaStream_t stream)
{
    const size_t smem = smem_bytes(D);
    const int threads = block_threads(D);
    // One block per SM has all the registers it asks for, two share the SM but spill.  Milliseconds,
    // one / two per SM: 300 modes 15.5 / 19.8 (72 rows) and 23.5 / 29.4 (143 rows); 512 modes up to
    // k = 10, 30.6 / 39.0; 600 modes 26.3 / 22.4 and 30.3 / 31.2; 1024 modes 43 / 34 and 52 / 38.
    const auto pick = [&](auto one, auto two, auto wide) {
        return threads > 256 ? wide : 2LL * n_modes <= 7LL * sms ? one : two;
    };
    const auto kernel = records ? pick(fwd_block_kernel<256, 1, true>, fwd_block_kernel<256, 2, true>,
                                       fwd_block_kernel<512, 1, true>)
                                : pick(fwd_block_kernel<256, 1, false>, fwd_block_kernel<256, 2, false>,
                                       fwd_block_kernel<512, 1, false>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DISCOEB_ECUDA;
    kernel<<<n_modes, threads, smem, stream>>>(cosmos, n_cosmo, mode_cosmo, ctrl, kmodes, tau_start, y0, sw, n_out,
                                        tau_out, D, y_full, y_out20, status, nsteps,
                                        records ? *records : StepRecords{}, gate);
    if (y_full) {
        const long long points = (long long)n_modes * n_out;
        project_states_kernel<<<(unsigned)((points + 3) / 4), 128, 0, stream>>>(cosmos, n_cosmo, mode_cosmo, points,
                                                                                kmodes, n_out, tau_out, D, status, y_full,
                                                                                y_out20);
    }
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

}  // namespace blk
}  // namespace dscb
