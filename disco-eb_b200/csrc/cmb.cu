// CMB source functions and the line-of-sight integral on sm_100a (include/discoeb.h).
//
// discoeb_sources: one warp per (mode, output time).  The warp re-evaluates the right-hand
//   side at the stored (RSA-projected) state, as compute_time_derivatives does
//   (perturbations.py:1339-1406), keeps y' in shared memory, and its leader assembles the
//   massive-neutrino moments, the Einstein-equation metric terms, the polarisation terms and
//   the Sachs-Wolfe, Doppler and polarisation sources of cmb.py:165-633 from them and from the
//   per-time background table.  y' never goes to HBM.  A second kernel (one thread per mode)
//   differentiates eta + alpha' along tau with a natural cubic spline (the ISW term) and sums S.
// discoeb_los: compute_theta_ell (cmb.py:680-835): optional spline resampling to a dense
//   log-k grid, spline resampling of every row onto the FFTLog log-chi grid with the bias
//   factor, a batched real-to-complex FFT in place (cuFFT), the coefficient table
//   M_l(p_n) = 2^(p-1) sqrt(pi) Gamma((1+l+p)/2) / Gamma((2+l-p)/2), and the contraction over
//   the frequencies as one FP64 GEMM on interleaved (re, im) pairs (cuBLAS): the complex sum
//   sum_n w_n Re(c_n k^-(p_n+1) M_l(p_n)) becomes a real dot product of length 2 n_freq.
// discoeb_cell: compute_Cell (cmb.py:838-873), trapezoid in ln k, one thread per l.
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "dgemm_i8.cuh"
#include "discoeb.h"
#include "fft_plans.cuh"
#include "lngamma.cuh"
#include "stepper.cuh"

using namespace dscb;
using namespace dscb::cplx;

namespace {

constexpr double kBias = -1.1;   // FFTLog bias (cmb.py:761)
constexpr double kPad = 2.0;     // padding of the log-chi range (cmb.py:738)

// ------------------------------------------------------------------------------------------
// sources

// Scalar parameters the source assembly reads: plain values, or values with their derivative
// along one parameter direction (DiscoebTangent) for the forward-mode sources.
template <class T> struct SrcPar {
    T grhom, Omegam, Omegab, OmegaDE, amnu, w0, wa;
};

// The source terms and their intermediates at one (mode, output time) from the state y, its
// time derivative yp and the background row bt[DISCOEB_BG_NFIELDS] (cmb.py:17-633), in the number
// type T: double for the sources, Dual for their derivative along a direction.  Y(i), YP(i) give
// the state and its derivative as T; out[DISCOEB_SRC_NFIELDS] (S and S1 are left to isw_kernel).
template <class T, class FY, class FYP>
__device__ void assemble_sources(const DiscoebCosmo& P, const SrcPar<T>& sp, const Dims& D, double k, const T* bt,
                                 FY Y, FYP YP, T* out)
{
    const int n = D.n;
    const T a = bt[DISCOEB_BG_A], aH = bt[DISCOEB_BG_APRIMEOA];
    const T rhonu = bt[DISCOEB_BG_RHONU], rho_Q = bt[DISCOEB_BG_RHO_Q];
    const T w_Q = bt[DISCOEB_BG_W_Q];
    const T opac = bt[DISCOEB_BG_OPAC], opacprime = bt[DISCOEB_BG_OPACPRIME];
    const T gvis = bt[DISCOEB_BG_GVIS], gvisprime = bt[DISCOEB_BG_GVISPRIME];
    const T gvispprime = bt[DISCOEB_BG_GVISPPRIME];
    // massive neutrinos (nu_perturb, nu_perturb_prime: perturbations.py:29-85; the derivative
    // of the speed is written as the reference writes it)
    T drhonu = 0.0, dpnu = 0.0, fnu = 0.0, shearnu = 0.0, rnp = 0.0, snp = 0.0;
    const int nq = D.nq, i0 = D.iq0, i1 = i0 + nq, i2 = i1 + nq;
    for (int q = 0; q < nq; ++q) {
        const T aq = a * sp.amnu / P.q[q];
        const T v = 1.0 / xsqrt(1.0 + aq * aq);
        const T vp = -0.5 * aq * aH * v * v * v;
        const double w = P.wq[q];
        drhonu += w * Y(i0 + q) / v;
        dpnu += w * Y(i0 + q) * v;
        fnu += w * Y(i1 + q);
        shearnu += w * Y(i2 + q) * v;
        rnp += w * (YP(i0 + q) / v - Y(i0 + q) / (v * v) * vp);
        snp += w * (YP(i2 + q) * v + Y(i2 + q) * vp);
    }
    dpnu = dpnu / 3.0;
    shearnu = shearnu * (2.0 / 3.0);
    snp = snp * (2.0 / 3.0);
    // metric (cmb.py:241-338)
    const int ig = 7, igp = D.idxgp, ir = D.idxr;
    const T eta = Y(2), deltac = Y(3), thetac = Y(4), deltab = Y(5), thetab = Y(6);
    const T deltag = Y(ig), thetag = Y(ig + 1), shearg = 0.5 * Y(ig + 2);
    const T deltar = Y(ir), thetar = Y(ir + 1), shearr = 0.5 * Y(ir + 2);
    const T deltaq = Y(n - 2), thetaq = Y(n - 1);
    const T thetabprime = YP(6), thetagprime = YP(ig + 1), sheargprime = 0.5 * YP(ig + 2);
    const T shearrprime = 0.5 * YP(ir + 2);
    const T a2 = a * a;
    const double k2 = k * k;
    const T Omegac = sp.Omegam - sp.Omegab;
    const T rpt = (1.0 + w_Q) * rho_Q * sp.grhom * sp.OmegaDE * thetaq * a2;
    const T grhoprime =
        (-sp.grhom * sp.Omegam / a - 2.0 * (P.grhog + P.grhor * (P.Neff + P.Nmnu * rhonu)) / a2 +
         sp.grhom * sp.OmegaDE * (-3.0 * (1.0 + sp.w0 + (1.0 - a) * sp.wa) * rho_Q * a2 + 2.0 * rho_Q * a2)) * aH +
        P.grhor * P.Nmnu * rnp / a2;
    const T aHprime = grhoprime / (6.0 * aH);
    const T dgrho = sp.grhom * (Omegac * deltac + sp.Omegab * deltab) / a +
                    (P.grhog * deltag + P.grhor * (P.Neff * deltar + P.Nmnu * drhonu)) / a2 +
                    sp.grhom * sp.OmegaDE * deltaq * rho_Q * a2;
    const T dgtheta = sp.grhom * (Omegac * thetac + sp.Omegab * thetab) / a +
                      4.0 / 3.0 * (P.grhog * thetag + P.Neff * P.grhor * thetar) / a2 +
                      P.Nmnu * P.grhor * k * fnu / a2 + rpt;
    const T dgshear = 4.0 / 3.0 * (P.grhog * shearg + P.Neff * P.grhor * shearr) / a2 +
                      P.Nmnu * P.grhor * shearnu / a2;
    const T dgshearprime = 4.0 / 3.0 * (P.grhog * sheargprime + P.Neff * P.grhor * shearrprime) / a2 +
                           P.Nmnu * P.grhor * snp / a2 - 2.0 * aH * dgshear;
    const T hprime = (2.0 * k2 * eta + dgrho) / aH;
    const T etaprime = 0.5 * dgtheta / k2;
    const T alpha = (hprime + 6.0 * etaprime) / 2.0 / k2;
    const T alphaprime = -3.0 * dgshear / (2.0 * k2) + eta - 2.0 * aH * alpha;
    const T alphapprime = -3.0 * dgshearprime / (2.0 * k2) + etaprime - 2.0 * (aHprime * alpha + aH * alphaprime);
    // polarisation (cmb.py:341-389)
    const T couplprime = 8.0 * (thetagprime + k2 * alphaprime) / 15.0 -
                         k * 0.6 * (YP(ig + 3) + YP(igp + 1) + YP(igp + 3));
    const T pol = Y(ig + 2) + Y(igp) + Y(igp + 2);
    const T polp = YP(ig + 2) + YP(igp) + YP(igp + 2);
    const T polpp = couplprime - 0.3 * (opacprime * pol + opac * polp);
    // sources (cmb.py:456-582); S1 needs d/dtau along the mode, see isw_kernel
    out[DISCOEB_SRC_S2] = gvis * (0.25 * deltag + 2.0 * alphaprime + pol / 16.0 + (thetabprime + 3.0 / 16.0 * polpp) / k2);
    out[DISCOEB_SRC_S3] = gvisprime * (alpha + (thetab + 3.0 / 8.0 * polp) / k2);
    out[DISCOEB_SRC_S4] = gvispprime * 3.0 / 16.0 * pol / k2;
    // E-mode polarisation source (3/4) g Pi of Zaldarriaga & Seljak (1997), whose Pi is a quarter
    // of pol (the reference's temperature terms Pi / 16, 3 Pi'' / 16 are theirs with that Pi)
    out[DISCOEB_SRC_E] = gvis * 3.0 / 16.0 * pol;
    out[DISCOEB_SRC_POTENTIAL] = eta + alphaprime;
    out[DISCOEB_SRC_ALPHA] = alpha;
    out[DISCOEB_SRC_ALPHAPRIME] = alphaprime;
    out[DISCOEB_SRC_ALPHAPPRIME] = alphapprime;
    out[DISCOEB_SRC_HPRIME] = hprime;
    out[DISCOEB_SRC_ETAPRIME] = etaprime;
    out[DISCOEB_SRC_APRIMEOAPRIME] = aHprime;
    out[DISCOEB_SRC_POL] = pol;
    out[DISCOEB_SRC_POLPRIME] = polp;
    out[DISCOEB_SRC_POLPPRIME] = polpp;
    out[DISCOEB_SRC_DRHONU] = drhonu;
    out[DISCOEB_SRC_DPNU] = dpnu;
    out[DISCOEB_SRC_FNU] = fnu;
    out[DISCOEB_SRC_SHEARNU] = shearnu;
    out[DISCOEB_SRC_RHONUPRIME] = rnp;
    out[DISCOEB_SRC_SHEARNUPRIME] = snp;
    out[DISCOEB_SRC_THETABPRIME] = thetabprime;
}

__global__ void __launch_bounds__(128) sources_kernel(const DiscoebCosmo* __restrict__ cosmo, int n_modes,
                                                      const double* __restrict__ kmodes, int n_tau,
                                                      const double* __restrict__ tau, const double* __restrict__ bt,
                                                      const double* __restrict__ y_full, double* fields)
{
    extern __shared__ double smem[];
    const int wib = threadIdx.x >> 5;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long n_points = (long long)n_modes * n_tau;
    if (warp >= n_points) return;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const DiscoebCosmo& P = *cosmo;
    const Dims D = make_dims(P);
    const int n = D.n;
    const int im = (int)(warp / n_tau), j = (int)(warp - (long long)im * n_tau);
    const double k = kmodes[im], t = tau[j];
    const double* y = y_full + (size_t)warp * n;
    double* yp = smem + (size_t)wib * n;
    Bg<double> b;
    bg_eval(P, y[0], t, k, -1, b);
    rhs_team(tm, P, D, b, k, t, y, yp, (double*)nullptr);
    tm.sync();
    if (!tm.leader()) return;
    double btj[DISCOEB_BG_NFIELDS];
    for (int f = 0; f < DISCOEB_BG_NFIELDS; ++f) btj[f] = bt[f * n_tau + j];
    const SrcPar<double> sp{P.grhom, P.Omegam, P.Omegab, P.OmegaDE, P.amnu, P.w0, P.wa};
    double out[DISCOEB_SRC_NFIELDS];
    assemble_sources(P, sp, D, k, btj, [&](int i) { return y[i]; }, [&](int i) { return yp[i]; }, out);
    const size_t stride = (size_t)n_points, o = (size_t)warp;
    for (int f = DISCOEB_SRC_S2; f < DISCOEB_SRC_NFIELDS; ++f) fields[f * stride + o] = out[f];
}

// The forward solve with the source assembly in its output stage: one warp per mode runs the
// adaptive solve (solve_mode) and, at each output time, projects the state (RSA), re-evaluates
// y' there and assembles the sources, exactly as discoeb_fwd followed by sources_kernel do, but
// without the full states going through HBM.  y_full (may be null) still receives the projected
// states.  Shared memory per warp: the cosmology and the mode's workspace.
constexpr int kCosmoDoublesC = (sizeof(DiscoebCosmo) + 7) / 8;

__global__ void __launch_bounds__(32) fwd_sources_kernel(
    const DiscoebCosmo* __restrict__ cosmo, DiscoebControl ctrl, int n_modes, const double* __restrict__ kmodes,
    const double* __restrict__ tau_start, const double* __restrict__ y0, const double* __restrict__ sw, int n_tau,
    const double* __restrict__ tau, const double* __restrict__ bt, int mem_doubles, double* y_full, double* fields,
    int32_t* status, int32_t* nsteps)
{
    extern __shared__ double smem[];
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const int mode = blockIdx.x;
    if (mode >= n_modes) return;
    DiscoebCosmo* P = reinterpret_cast<DiscoebCosmo*>(smem);
    double* wmem = smem + kCosmoDoublesC;
    {
        const int* src = reinterpret_cast<const int*>(cosmo);
        int* dst = reinterpret_cast<int*>(P);
        for (int i = tm.lane; i < (int)(sizeof(DiscoebCosmo) / 4); i += 32) dst[i] = src[i];
    }
    tm.sync();
    const Dims D = make_dims(*P);
    const int n = D.n;
    const size_t stride = (size_t)n_modes * n_tau;
    const double qnan = __longlong_as_double(0x7ff8000000000000LL);
    auto fill_nan = [&](int from) {
        for (int j = from; j < n_tau; ++j) {
            const size_t o = (size_t)mode * n_tau + j;
            for (int f = tm.lane; f < DISCOEB_SRC_NFIELDS; f += 32) fields[f * stride + o] = qnan;
            if (y_full)
                for (int i = tm.lane; i < n; i += 32) y_full[o * n + i] = qnan;
        }
    };
    if (mode_mem_doubles(D) != mem_doubles) {
        fill_nan(0);
        if (tm.leader()) {
            status[mode] = DISCOEB_BAD_INDEX;
            nsteps[mode] = 0;
        }
        return;
    }
    ModeMem M = carve(wmem, D);
    const double k = kmodes[mode];
    for (int i = tm.lane; i < n; i += 32) M.y[i] = y0[(size_t)mode * n + i];
    const double swm[3] = {sw[3 * mode], sw[3 * mode + 1], sw[3 * mode + 2]};
    tm.sync();
    const SrcPar<double> sp{P->grhom, P->Omegam, P->Omegab, P->OmegaDE, P->amnu, P->w0, P->wa};
    auto emit = [&](int j, const double* y, int) {
        const double t = tau[j];
        // the projected state into M.f, y' there into M.dT (both are rebuilt at the next step start)
        double fld[4];
        const bool rsa = rsa_projection<double>(*P, nullptr, D, t, k, y, nullptr, fld);
        const size_t o = (size_t)mode * n_tau + j;
        for (int i = tm.lane; i < n; i += 32) {
            double v = y[i];
            if (rsa) {
                const int sl = rsa_slot(D, i);
                if (sl >= 0) v = fld[sl];
                else if (sl == -1) v = 0.0;
            }
            M.f[i] = v;
            if (y_full) y_full[o * n + i] = v;
        }
        tm.sync();
        Bg<double> b;
        bg_eval(*P, M.f[0], t, k, -1, b);
        rhs_team(tm, *P, D, b, k, t, M.f, M.dT, (double*)nullptr);
        tm.sync();
        if (tm.leader()) {
            double btj[DISCOEB_BG_NFIELDS];
            for (int f = 0; f < DISCOEB_BG_NFIELDS; ++f) btj[f] = bt[f * n_tau + j];
            double out[DISCOEB_SRC_NFIELDS];
            assemble_sources(*P, sp, D, k, btj, [&](int i) { return M.f[i]; }, [&](int i) { return M.dT[i]; }, out);
            for (int f = DISCOEB_SRC_S2; f < DISCOEB_SRC_NFIELDS; ++f) fields[f * stride + o] = out[f];
        }
        tm.sync();
    };
    const SolveResult R = solve_mode(tm, *P, D, ctrl, k, tau_start[mode], swm, n_tau, tau, M, emit);
    fill_nan(R.outputs);
    if (tm.leader()) {
        status[mode] = R.status;
        nsteps[mode] = R.steps;
    }
}

// Natural cubic spline second derivatives through (x[i], y[i*ys]) for i < n (the Thomas
// recurrence of spline_interpolation.py:19-75), written to S[i*ys]; cp is scratch of n
// doubles with stride cs.
__device__ void spline_second(int n, const double* x, int xs, const double* y, long long ys, double* S, double* cp,
                              long long cs)
{
    S[0] = 0.0;
    S[(long long)(n - 1) * ys] = 0.0;
    const int m = n - 2;
    if (m <= 0) return;
    auto X = [&](int i) { return x[(long long)i * xs]; };
    auto Y = [&](int i) { return y[(long long)i * ys]; };
    // forward sweep: cp in cp[], dp in S[1..]
    double dprev = 0.0, cprev = 0.0;
    for (int i = 0; i < m; ++i) {
        const double h0 = X(i + 1) - X(i), h1 = X(i + 2) - X(i + 1);
        const double a = h0, bb = 2.0 * (h0 + h1), c = h1;
        const double d = 6.0 * ((Y(i + 2) - Y(i + 1)) / h1 - (Y(i + 1) - Y(i)) / h0);
        double cc, dd;
        if (i == 0) {
            cc = c / bb;
            dd = d / bb;
        } else {
            const double den = bb - a * cprev;
            cc = (i < m - 1) ? c / den : 0.0;
            dd = (d - a * dprev) / den;
        }
        cp[(long long)i * cs] = cc;
        S[(long long)(i + 1) * ys] = dd;
        cprev = cc;
        dprev = dd;
    }
    for (int i = m - 2; i >= 0; --i)
        S[(long long)(i + 1) * ys] = S[(long long)(i + 1) * ys] - cp[(long long)i * cs] * S[(long long)(i + 2) * ys];
}

// interval index of the reference: count(x < xn) - 1, clipped to [0, n-2]
__device__ int spline_interval(const double* x, int xs, int n, double xn)
{
    int lo = 0, hi = n;  // first index with x >= xn
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x[(long long)mid * xs] < xn) lo = mid + 1;
        else hi = mid;
    }
    int i = lo - 1;
    if (i < 0) i = 0;
    if (i > n - 2) i = n - 2;
    return i;
}

__device__ double spline_value(double x0, double x1, double y0, double y1, double S0, double S1, double xn)
{
    const double h = x1 - x0, t = (xn - x0) / h, A = 1.0 - t, B = t;
    return A * y0 + B * y1 + ((A * A * A - A) * S0 + (B * B * B - B) * S1) * (h * h) / 6.0;
}

__device__ double spline_slope(double x0, double x1, double y0, double y1, double S0, double S1, double xn)
{
    const double h = x1 - x0, d = xn - x0;
    const double b = (y1 - y0) / h - h * (S1 + 2.0 * S0) / 6.0, c = S0 / 2.0, dd = (S1 - S0) / (6.0 * h);
    return b + 2.0 * c * d + 3.0 * dd * d * d;
}

// S1 = exp(-optical depth) d(eta + alpha')/dtau with a natural spline along tau per mode
// (compute_source_term_isw, cmb.py:392-453), S = S1 + S2 + S3 + S4.  A block per mode: one thread runs
// the spline's recurrence, all of them the slopes (a binary search each, most of the time when one
// thread had them all: 128 modes 0.67 -> 0.13 ms).
__global__ void __launch_bounds__(64) isw_kernel(int n_modes, int n_tau, const double* __restrict__ tau,
                                                 const double* __restrict__ bt, double* fields, double* scratch)
{
    const int im = blockIdx.x;
    const size_t stride = (size_t)n_modes * n_tau, row = (size_t)im * n_tau;
    const double* pot = fields + DISCOEB_SRC_POTENTIAL * stride + row;
    double* S1 = fields + DISCOEB_SRC_S1 * stride + row;  // holds the second derivatives first
    double* cp = scratch + row;
    if (threadIdx.x == 0) spline_second(n_tau, tau, 1, pot, 1, S1, cp, 1);
    __syncthreads();
    for (int j = threadIdx.x; j < n_tau; j += blockDim.x) {
        const int i = spline_interval(tau, 1, n_tau, tau[j]);
        cp[j] = spline_slope(tau[i], tau[i + 1], pot[i], pot[i + 1], S1[i], S1[i + 1], tau[j]);
    }
    __syncthreads();
    double* S = fields + DISCOEB_SRC_S * stride + row;
    const double* S2 = fields + DISCOEB_SRC_S2 * stride + row;
    const double* S3 = fields + DISCOEB_SRC_S3 * stride + row;
    const double* S4 = fields + DISCOEB_SRC_S4 * stride + row;
    for (int j = threadIdx.x; j < n_tau; j += blockDim.x) {
        const double s1 = exp(-bt[DISCOEB_BG_OPTICAL_DEPTH * n_tau + j]) * cp[j];
        S1[j] = s1;
        S[j] = s1 + S2[j] + S3[j] + S4[j];
    }
}

// ------------------------------------------------------------------------------------------
// line of sight

// lo = ln chi_min - 2, dl = (ln chi_max + 2 - lo) / n_fft of compute_theta_ell (cmb.py:730-745)
__global__ void geom_kernel(int n_tau, const double* __restrict__ tau, double tau0, int n_fft, double* g)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const double chi_min = fmax(tau0 - tau[n_tau - 1], 1.0), chi_max = tau0 - tau[0];
    const double lo = log(chi_min) - kPad, hi = log(chi_max) + kPad;
    g[0] = lo;
    g[1] = (hi - lo) / n_fft;
}

// spline second derivatives along ln k for every tau column (one thread per column)
__global__ void k_spline_log_kernel(int n_modes, const double* __restrict__ lk, int n_tau, const double* S, double* S2k,
                                    double* cp)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_tau) return;
    spline_second(n_modes, lk, 1, S + j, n_tau, S2k + j, cp + j, n_tau);
}

__global__ void log_kernel(int n, const double* __restrict__ x, double* lx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) lx[i] = log(x[i]);
}

// S on the dense log-k grid: Sd[kd, j]; also the dense k values
__global__ void k_dense_kernel(int n_modes, const double* __restrict__ lk, int n_tau, const double* __restrict__ S,
                               const double* __restrict__ S2k, int n_dense, double* Sd, double* kd)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_dense * n_tau) return;
    const int id = (int)(t / n_tau), j = (int)(t - (long long)id * n_tau);
    const double lk0 = lk[0], lk1 = lk[n_modes - 1];
    const double x = (id == n_dense - 1) ? lk1 : lk0 + id * ((lk1 - lk0) / (n_dense - 1));
    const int i = spline_interval(lk, 1, n_modes, x);
    const size_t r0 = (size_t)i * n_tau + j, r1 = r0 + n_tau;
    Sd[t] = spline_value(lk[i], lk[i + 1], S[r0], S[r1], S2k[r0], S2k[r1], x);
    if (j == 0) kd[id] = exp(x);
}

// per-row spline second derivatives along ln chi (chi = tau0 - tau, increasing), one thread per row
__global__ void chi_spline_kernel(int n_rows, int n_tau, const double* __restrict__ lchi, const double* Srow,
                                  double* S2c, double* cp)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    // row values in chi order: S[r, n_tau - 1 - m]
    const double* y = Srow + (size_t)r * n_tau + (n_tau - 1);
    spline_second(n_tau, lchi, 1, y, -1, S2c + (size_t)r * n_tau + (n_tau - 1), cp + (size_t)r * n_tau, 1);
}

// ln chi of the knots, chi = tau0 - tau in increasing order (cmb.py:724-752)
__global__ void lchi_kernel(int n_tau, const double* __restrict__ tau, double tau0, double* lchi)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_tau) lchi[t] = log(fmax(tau0 - tau[n_tau - 1 - t], 1e-10));
}

// per FFTLog point: interval index among the knots, abscissa ln chi_m, and chi_m^-bias
__global__ void fgrid_kernel(int n_tau, const double* __restrict__ lchi, int n_fft, const double* __restrict__ g,
                             int* fidx, double* fx, double* fbias)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_fft) return;
    const double cf = exp(g[0] + t * g[1]);
    const double x = log(cf);
    fidx[t] = spline_interval(lchi, 1, n_tau, x);
    fx[t] = x;
    fbias[t] = pow(cf, -kBias);
}

// biased source on the FFTLog grid into the in-place FFT buffer (row pitch `pitch` doubles)
__global__ void chi_eval_kernel(int n_rows, int n_tau, const double* __restrict__ lchi, const double* __restrict__ Srow,
                                const double* __restrict__ S2c, int n_fft, const int* __restrict__ fidx,
                                const double* __restrict__ fx, const double* __restrict__ fbias, long long pitch,
                                double* F)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n_fft) return;
    const int i = fidx[m];
    // the point's weights (spline_value), formed once for its rows: 0.70 -> 0.37 ms for 8192 rows of 16384
    const double fb = fbias[m], l0 = lchi[i], h = lchi[i + 1] - l0, B = (fx[m] - l0) / h, A = 1.0 - B, hh = h * h / 6.0 * fb;
    const double w0 = A * fb, w1 = B * fb, w2 = (A * A * A - A) * hh, w3 = (B * B * B - B) * hh;
    for (int r = blockIdx.y; r < n_rows; r += gridDim.y) {
        const size_t base = (size_t)r * n_tau + (n_tau - 1);
        F[(size_t)r * pitch + m] = w0 * Srow[base - i] + w1 * Srow[base - i - 1] +
                                   (w2 * S2c[base - i] + w3 * S2c[base - i - 1]);
    }
}

// e^{-i eta (lo + ln k)} along a row of frequencies eta = c0 q, q = thread, thread + kPhaseThreads, ...:
// one sine and cosine per thread and row, then a rotation per frequency (a sine, a cosine, an
// exponential and a logarithm per element bound the kernel: 8192 rows of 8193, 0.69 -> 0.39 ms).  The
// error of the angle is max(|phase|, number of rotations) 2^-53: rotations add one each, which matters
// only where the phase itself is small, and there it is n_fft / 512 2^-53
constexpr int kPhaseThreads = 256;
struct PhaseWalk {
    double lk, mag, sn, cs, rs, rc;
    __device__ PhaseWalk(double k, double lo, double c0, int n_fft)
    {
        lk = log(k);
        mag = exp(-(kBias + 1.0) * lk) / n_fft;
        const double th = -c0 * (lo + lk);
        sincos(th * (double)threadIdx.x, &sn, &cs);
        sincos(th * (double)kPhaseThreads, &rs, &rc);
    }
    __device__ void step()
    {
        const double s = sn * rc + cs * rs;
        cs = cs * rc - sn * rs;
        sn = s;
    }
};

// c_n k^-(p_n+1) with the rfft normalisation and the interval phase, times the weight of the
// real reconstruction (1 for n = 0 and the Nyquist term, 2 otherwise), in place
__global__ void ck_kernel(int n_rows, const double* __restrict__ krow, int n_fft, int n_freq,
                          const double* __restrict__ g, long long pitch, double* F)
{
    const double lo = g[0], c0 = 2.0 * M_PI / (n_fft * g[1]);  // eta = c0 q
    for (int r = blockIdx.x; r < n_rows; r += gridDim.x) {
        PhaseWalk ph(krow[r], lo, c0, n_fft);
        for (int q = threadIdx.x; q < n_freq; q += kPhaseThreads, ph.step()) {
            const double mag = (q == 0 || ((n_fft % 2 == 0) && q == n_freq - 1)) ? ph.mag : 2.0 * ph.mag;
            double* c = F + (size_t)r * pitch + 2 * q;
            const double re = c[0], im = c[1];
            c[0] = mag * (re * ph.cs - im * ph.sn);
            c[1] = mag * (re * ph.sn + im * ph.cs);
        }
    }
}

// B[l, 2q] = Re M_l(p_q), B[l, 2q + 1] = -Im M_l(p_q) (cmb.py:636-677)
// One thread per (frequency, run of kMcoefRun multipoles of one parity): log-Gamma at the run's
// first l, the recurrence in l + 2 after it (fftlog_mcoef_run).  Threads with consecutive
// frequencies write consecutive 16-byte (re, im) pairs of a row.  gd / Bd (may be null): the
// table's derivative along the spacing's derivative gd[1].
constexpr int kMcoefRun = 16;

__global__ void mcoef_kernel(int n_ell, int n_freq, int n_fft, const double* __restrict__ g,
                             const double* __restrict__ gd, double* B, double* Bd)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long runs = 2LL * ((n_ell + 2 * kMcoefRun - 1) / (2 * kMcoefRun));
    if (t >= runs * n_freq) return;
    const int q = (int)(t % n_freq);
    const long long r = t / n_freq;
    const int l0 = (int)(r & 1) + 2 * kMcoefRun * (int)(r >> 1);
    if (l0 >= n_ell) return;
    const int count = min(kMcoefRun, (n_ell - 1 - l0) / 2 + 1);
    const size_t o = (size_t)l0 * (2 * (size_t)n_freq) + 2 * q;
    const long long step = 4LL * n_freq;
    double* Bo = B ? B + o : nullptr;
    double* Bdo = Bd ? Bd + o : nullptr;
    const double dl_dot = gd ? gd[1] : 0.0;
    if (l0 < 2) {
        // l = 0, 1: the log-Gamma of (1 + l + p)/2 takes its reflection branch, which overflows to
        // M = 0 at large eta as the reference's does; evaluated directly, the run starts at l0 + 2
        double b[2], bd[2];
        fftlog_mcoef(l0, q, n_fft, kBias, g[1], dl_dot, b, Bdo ? bd : nullptr);
        if (Bo) Bo[0] = b[0], Bo[1] = b[1];
        if (Bdo) Bdo[0] = bd[0], Bdo[1] = bd[1];
        if (count > 1)
            fftlog_mcoef_run(l0 + 2, count - 1, q, n_fft, kBias, g[1], dl_dot, step, Bo ? Bo + step : nullptr,
                             Bdo ? Bdo + step : nullptr);
        return;
    }
    fftlog_mcoef_run(l0, count, q, n_fft, kBias, g[1], dl_dot, step, Bo, Bdo);
}

long long mcoef_threads(int n_ell, int n_freq)
{
    return 2LL * ((n_ell + 2 * kMcoefRun - 1) / (2 * kMcoefRun)) * n_freq;
}

// C_l = trapezoid over ln k of (k/k_p)^(n_s-1) Theta_l(k)^2, written as sum_i w_i Theta_il^2 with
// w_i = (k_i/k_p)^(n_s-1) (ln k_{i+1} - ln k_{i-1})/2 (one-sided at the ends).  A block owns 32
// consecutive l (one coalesced 256-byte row segment per mode) and its 8 warps stride over the
// modes; the weights of a chunk of modes are computed once per block into shared memory.
constexpr int kCellChunk = 1024;

// trapezoid weight in ln k of mode i times the primordial factor (k_i/k_p)^(n_s-1)
__device__ inline double cell_weight(int i, int n_modes, const double* __restrict__ kmodes, double n_s, double k_p)
{
    const double lk = log(kmodes[i]);
    const double lo = i > 0 ? log(kmodes[i - 1]) : lk;
    const double hi = i + 1 < n_modes ? log(kmodes[i + 1]) : lk;
    return pow(kmodes[i] / k_p, n_s - 1.0) * (0.5 * (hi - lo));
}

__global__ void __launch_bounds__(256) cell_kernel(int n_modes, const double* __restrict__ kmodes, int n_ell,
                                                   const double* __restrict__ theta, double n_s, double k_p,
                                                   double* cell, bool d_n_s = false,
                                                   const double* __restrict__ theta_b = nullptr)
{
    __shared__ double w[kCellChunk];
    __shared__ double part[8][32];
    const int lx = threadIdx.x & 31, wy = threadIdx.x >> 5;
    const int l = blockIdx.x * 32 + lx;
    double acc = 0.0;
    for (int c0 = 0; c0 < n_modes; c0 += kCellChunk) {
        const int cn = min(kCellChunk, n_modes - c0);
        __syncthreads();
        // d_n_s: the weights' derivative in n_s, ln(k_i/k_p) w_i, for d C_l / d n_s
        for (int j = threadIdx.x; j < cn; j += blockDim.x)
            w[j] = cell_weight(c0 + j, n_modes, kmodes, n_s, k_p) * (d_n_s ? log(kmodes[c0 + j] / k_p) : 1.0);
        __syncthreads();
        if (l < n_ell) {
#pragma unroll 4
            for (int j = wy; j < cn; j += 8) {
                const double th = theta[(size_t)(c0 + j) * n_ell + l];
                const double tb = theta_b ? theta_b[(size_t)(c0 + j) * n_ell + l] : th;  // cross spectrum
                acc += w[j] * (th * tb);
            }
        }
    }
    part[wy][lx] = acc;
    __syncthreads();
    if (wy == 0 && l < n_ell) {
        double sum = 0.0;
        for (int q = 0; q < 8; ++q) sum += part[q][lx];
        cell[l] = sum;
    }
}

// ------------------------------------------------------------------------------------------
// E-mode line of sight: Theta_E,l(k) = sqrt((l+2)!/(l-2)!) int S_E(k, tau) j_l(x) / x^2 dtau,
// x = k (tau0 - tau) (Zaldarriaga & Seljak 1997).  Below kELSwitch: the FFTLog integral of
// S_E / chi^2 (chi held >= 1 Mpc: S_E ~ 0 today, where 1/chi^2 diverges) times the factor / k^2.
// From kELSwitch on, where that integral's absolute FFTLog error times l^2 / k^2 would swamp the
// signal: j_l / x^2 = [j_{l-2} / (2l-1) + j_l (1/(2l-1) + 1/(2l+3)) + j_{l+2} / (2l+3)] / (2l+1)
// (from j_{l-1} + j_{l+1} = (2l+1) j_l / x), i.e. the FFTLog integrals of S_E itself at l - 2, l,
// l + 2 with positive weights (no cancellation).  Below l = 4 the recurrence would need
// l - 2 < 2, outside the FFTLog's convergence strip at bias -1.1.
constexpr int kELSwitch = 8;

__device__ __forceinline__ double e_factor(int l)
{
    return l >= 2 ? sqrt((l + 2.0) * (l + 1.0) * l * (l - 1.0)) : 0.0;
}

__global__ void e_source_kernel(int n_modes, int n_tau, const double* __restrict__ tau, double tau0,
                                const double* __restrict__ S, double* out)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_modes * n_tau) return;
    const int j = (int)(t % n_tau);
    const double chi = fmax(tau0 - tau[j], 1.0);
    out[t] = S[t] / (chi * chi);
}

// theta[r, l] for l < nlo from the direct integrals th_lo [rows, nlo]
__global__ void e_low_kernel(int rows, int n_ell, int nlo, const double* __restrict__ k,
                             const double* __restrict__ th_lo, double* theta)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)rows * nlo) return;
    const int r = (int)(t / nlo), l = (int)(t - (long long)r * nlo);
    theta[(size_t)r * n_ell + l] = th_lo[t] * e_factor(l) / (k[r] * k[r]);
}

// theta[r, l] for nlo <= l < n_ell from the integrals of S_E th [rows, n_ell + 2] by the recurrence
__global__ void e_high_kernel(int rows, int n_ell, int nlo, const double* __restrict__ th, double* theta)
{
    const int span = n_ell - nlo;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (span <= 0 || t >= (long long)rows * span) return;
    const int r = (int)(t / span), l = nlo + (int)(t - (long long)r * span);
    const double* row = th + (size_t)r * (n_ell + 2);
    const double a = 2.0 * l + 1.0, cm = 1.0 / (a * (2.0 * l - 1.0)), cp = 1.0 / (a * (2.0 * l + 3.0));
    theta[(size_t)r * n_ell + l] = e_factor(l) * (cm * row[l - 2] + (cm + cp) * row[l] + cp * row[l + 2]);
}

// ------------------------------------------------------------------------------------------
// tangent of C_l along one direction of the line of sight's inputs (sources S', output times
// tau', tau0'): forward mode through the resampling, the FFT coefficients and the table M_l(p),
// folded into C_l = sum_k w_k Theta_kl^2 with Theta = A B^T (A the coefficient rows, B the
// table): dC_l = 2 sum_j (B_lj H_lj + B'_lj G_lj), G = Omega^T A, H = Omega^T A',
// Omega_kl = w_k Theta_kl.  The interval indices of the resampling are those of the base point.

// d(lo, dl) of geom_kernel's grid: it moves with tau0 - tau at the last and first knots
__global__ void geom_dot_kernel(int n_tau, const double* __restrict__ tau, const double* __restrict__ tau_dot,
                                double tau0, double tau0_dot, int n_fft, double* gd)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const double cmin = tau0 - tau[n_tau - 1];
    const double lo_dot = cmin > 1.0 ? (tau0_dot - tau_dot[n_tau - 1]) / cmin : 0.0;  // else held by fmax
    const double hi_dot = (tau0_dot - tau_dot[0]) / (tau0 - tau[0]);
    gd[0] = lo_dot;
    gd[1] = (hi_dot - lo_dot) / n_fft;
}

// d ln chi of the knots (lchi_kernel)
__global__ void lchi_dot_kernel(int n_tau, const double* __restrict__ tau, const double* __restrict__ tau_dot,
                                double tau0, double tau0_dot, double* lchi_dot)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tau) return;
    const double c = tau0 - tau[n_tau - 1 - t];
    lchi_dot[t] = c > 1e-10 ? (tau0_dot - tau_dot[n_tau - 1 - t]) / c : 0.0;
}

// d ln chi_m and d chi_m^-bias of the FFTLog points (fgrid_kernel: ln chi_m = lo + m dl)
__global__ void fgrid_dot_kernel(int n_fft, const double* __restrict__ gd, const double* __restrict__ fbias,
                                 double* fx_dot, double* fbias_dot)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_fft) return;
    const double xd = gd[0] + t * gd[1];
    fx_dot[t] = xd;
    fbias_dot[t] = -kBias * xd * fbias[t];
}

// spline_second in dual numbers: knots x + e x', values y + e y' (value stride ys, knot stride 1);
// the second derivatives' values and derivatives go to S, S_dot (stride ys); cp, cp_dot scratch
__device__ void spline_second_dual(int n, const double* x, const double* xd, const double* y, const double* yd,
                                   long long ys, double* S, double* Sd, double* cp, double* cpd)
{
    S[0] = Sd[0] = 0.0;
    S[(long long)(n - 1) * ys] = Sd[(long long)(n - 1) * ys] = 0.0;
    const int m = n - 2;
    if (m <= 0) return;
    auto X = [&](int i) { return Dual(x[i], xd[i]); };
    auto Y = [&](int i) { return Dual(y[(long long)i * ys], yd[(long long)i * ys]); };
    Dual dprev(0.0), cprev(0.0);
    for (int i = 0; i < m; ++i) {
        const Dual h0 = X(i + 1) - X(i), h1 = X(i + 2) - X(i + 1);
        const Dual a = h0, bb = 2.0 * (h0 + h1), c = h1;
        const Dual d = 6.0 * ((Y(i + 2) - Y(i + 1)) / h1 - (Y(i + 1) - Y(i)) / h0);
        Dual cc, dd;
        if (i == 0) {
            cc = c / bb;
            dd = d / bb;
        } else {
            const Dual den = bb - a * cprev;
            cc = (i < m - 1) ? c / den : Dual(0.0);
            dd = (d - a * dprev) / den;
        }
        cp[i] = cc.v;
        cpd[i] = cc.d;
        S[(long long)(i + 1) * ys] = dd.v;
        Sd[(long long)(i + 1) * ys] = dd.d;
        cprev = cc;
        dprev = dd;
    }
    for (int i = m - 2; i >= 0; --i) {
        const long long a1 = (long long)(i + 1) * ys, a2 = (long long)(i + 2) * ys;
        const Dual r = Dual(S[a1], Sd[a1]) - Dual(cp[i], cpd[i]) * Dual(S[a2], Sd[a2]);
        S[a1] = r.v;
        Sd[a1] = r.d;
    }
}

// chi_spline_kernel in dual numbers (one thread per row; rows in chi order as there)
__global__ void chi_spline_dot_kernel(int n_rows, int n_tau, const double* __restrict__ lchi,
                                      const double* __restrict__ lchi_dot, const double* Srow, const double* Srow_dot,
                                      double* S2v, double* S2d, double* cpv, double* cpd)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rows) return;
    const size_t last = (size_t)r * n_tau + (n_tau - 1);
    spline_second_dual(n_tau, lchi, lchi_dot, Srow + last, Srow_dot + last, -1, S2v + last, S2d + last,
                       cpv + (size_t)r * n_tau, cpd + (size_t)r * n_tau);
}

// the derivative of chi_eval_kernel's biased source on the FFTLog grid, into F_dot (row pitch)
__global__ void chi_eval_dot_kernel(int n_rows, int n_tau, const double* __restrict__ lchi,
                                    const double* __restrict__ lchi_dot, const double* __restrict__ Srow,
                                    const double* __restrict__ Srow_dot, const double* __restrict__ S2v,
                                    const double* __restrict__ S2d, int n_fft, const int* __restrict__ fidx,
                                    const double* __restrict__ fx, const double* __restrict__ fx_dot,
                                    const double* __restrict__ fbias, const double* __restrict__ fbias_dot,
                                    long long pitch, double* Fd)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n_fft) return;
    const int i = fidx[m];
    const Dual l0(lchi[i], lchi_dot[i]), l1(lchi[i + 1], lchi_dot[i + 1]), x(fx[m], fx_dot[m]);
    const Dual fb(fbias[m], fbias_dot[m]);
    const Dual h = l1 - l0, B = (x - l0) / h, A = 1.0 - B, hh = h * h / 6.0 * fb;
    const Dual w0 = A * fb, w1 = B * fb, w2 = (A * A * A - A) * hh, w3 = (B * B * B - B) * hh;
    for (int r = blockIdx.y; r < n_rows; r += gridDim.y) {
        const size_t p0 = (size_t)r * n_tau + (n_tau - 1) - i, p1 = p0 - 1;
        Fd[(size_t)r * pitch + m] = (w0.v * Srow_dot[p0] + w1.v * Srow_dot[p1] + (w2.v * S2d[p0] + w3.v * S2d[p1])) +
                                    (w0.d * Srow[p0] + w1.d * Srow[p1] + (w2.d * S2v[p0] + w3.d * S2v[p1]));
    }
}

// the derivative of ck_kernel's coefficients: c = mag e^{i ph} F with ph = -eta (lo + ln k) and
// eta = 2 pi q / (n_fft dl), so c' = mag e^{i ph} F' + i ph' c; Fd holds F' (the FFT of the
// derivative rows) and becomes c', C holds the base point's c
__global__ void ck_dot_kernel(int n_rows, const double* __restrict__ krow, int n_fft, int n_freq,
                              const double* __restrict__ g, const double* __restrict__ gd, long long pitch,
                              const double* __restrict__ C, double* Fd)
{
    const double lo = g[0], dl = g[1], c0 = 2.0 * M_PI / (n_fft * dl);  // eta = c0 q
    for (int r = blockIdx.x; r < n_rows; r += gridDim.x) {
        PhaseWalk ph(krow[r], lo, c0, n_fft);
        const double ph1 = -c0 * (gd[0] - gd[1] / dl * (lo + ph.lk));  // d phase per q
        for (int q = threadIdx.x; q < n_freq; q += kPhaseThreads, ph.step()) {
            const double mag = (q == 0 || ((n_fft % 2 == 0) && q == n_freq - 1)) ? ph.mag : 2.0 * ph.mag;
            const double ph_dot = ph1 * q;
            const size_t o = (size_t)r * pitch + 2 * q;
            const double re = Fd[o], im = Fd[o + 1];
            Fd[o] = mag * (re * ph.cs - im * ph.sn) - ph_dot * C[o + 1];
            Fd[o + 1] = mag * (re * ph.sn + im * ph.cs) + ph_dot * C[o];
        }
    }
}

__global__ void cell_weight_kernel(int n_modes, const double* __restrict__ kmodes, double n_s, double k_p, double* w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_modes) w[i] = cell_weight(i, n_modes, kmodes, n_s, k_p);
}

// Omega_kl = w_k Theta_kl in place
__global__ void scale_rows_kernel(int n_rows, int n_cols, const double* __restrict__ w, double* M)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_rows * n_cols) return;
    M[t] *= w[t / n_cols];
}

// dC_l = 2 sum_j (B_lj H_lj + Bd_lj G_lj): one block per l, rows of `pitch` doubles
__global__ void __launch_bounds__(256) cell_dot_kernel(int n_ell, long long pitch, const double* __restrict__ B,
                                                       const double* __restrict__ H, const double* __restrict__ Bd,
                                                       const double* __restrict__ G, double* out)
{
    __shared__ double part[256];
    const int l = blockIdx.x;
    if (l >= n_ell) return;
    const size_t o = (size_t)l * pitch;
    double acc = 0.0;
    for (long long j = threadIdx.x; j < pitch; j += blockDim.x) acc += B[o + j] * H[o + j] + Bd[o + j] * G[o + j];
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[l] = 2.0 * part[0];
}

// ------------------------------------------------------------------------------------------
// forward-mode sources: the derivative of S along one parameter direction from the states' and
// output times' derivatives, the tables' (DiscoebTangent) and the background rows' derivatives

// one warp per (direction, mode, output time): y' and its derivative (the e-part of f at
// y + e y_dot under the dual background, plus d f / d tau at fixed y times tau_dot), then the
// assembly in dual numbers; writes the derivatives of S2, S3, S4 and the potential eta + alpha'
__global__ void __launch_bounds__(128) sources_dot_kernel(
    const DiscoebCosmo* __restrict__ cosmo, const DiscoebTangent* __restrict__ tangents, int n_dir, int n_modes,
    const double* __restrict__ kmodes, int n_tau, const double* __restrict__ tau, const double* __restrict__ tau_dot,
    const double* __restrict__ bt, const double* __restrict__ bt_dot, const double* __restrict__ y_full,
    const double* __restrict__ y_full_dot, double* fd4, double* se_dot)
{
    extern __shared__ double smem[];
    const int wib = threadIdx.x >> 5;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long n_points = (long long)n_modes * n_tau;
    if (warp >= n_points) return;
    const WarpTeam tm{(int)(threadIdx.x & 31)};
    const DiscoebCosmo& P = *cosmo;
    const Dims D = make_dims(P);
    const int n = D.n;
    const long long pt = warp;
    const int im = (int)(pt / n_tau), j = (int)(pt - (long long)im * n_tau);
    const double k = kmodes[im], t = tau[j];
    const double* y = y_full + (size_t)pt * n;
    double* yp = smem + (size_t)wib * 2 * n;
    double* ypd = yp + n;
    // the base point's y' once per point, then each direction's derivative part
    Bg<double> b;
    bg_eval(P, y[0], t, k, -1, b);
    rhs_team(tm, P, D, b, k, t, y, yp, (double*)nullptr);
    int hint = P.xe_loga.n_knots / 2;
    const size_t stride = (size_t)n_dir * n_points;
    for (int d = 0; d < n_dir; ++d) {
        const DiscoebTangent* TN = tangents + d;
        const double tdot = tau_dot[(size_t)d * n_tau + j];
        const double* yd = y_full_dot + ((size_t)d * n_points + pt) * n;
        Bg<Dual> bd;
        bg_eval_team(tm, P, Dual(y[0], yd[0]), t, k, -1, bd, hint, TN);
        rhs_team(tm, P, D, bd, k, t, y, ypd, (double*)nullptr, yd, (const double*)nullptr, 1, 1);
        tm.sync();
        for (int i = tm.lane; i < n; i += 32) ypd[i] += dtau_row(D, b, t, i, y) * tdot;
        tm.sync();
        if (tm.leader()) {
            Dual btj[DISCOEB_BG_NFIELDS];
            for (int f = 0; f < DISCOEB_BG_NFIELDS; ++f)
                btj[f] = Dual(bt[f * n_tau + j], bt_dot[((size_t)d * DISCOEB_BG_NFIELDS + f) * n_tau + j]);
            const SrcPar<Dual> sp{Dual(P.grhom, TN->grhom), Dual(P.Omegam, TN->Omegam),
                                  Dual(P.Omegab, TN->Omegab), Dual(P.OmegaDE, TN->OmegaDE),
                                  Dual(P.amnu, TN->amnu),   Dual(P.w0, TN->w0),
                                  Dual(P.wa, TN->wa)};
            Dual out[DISCOEB_SRC_NFIELDS];
            assemble_sources(P, sp, D, k, btj, [&](int i) { return Dual(y[i], yd[i]); },
                             [&](int i) { return Dual(yp[i], ypd[i]); }, out);
            const size_t o = (size_t)d * n_points + pt;
            fd4[0 * stride + o] = out[DISCOEB_SRC_S2].d;
            fd4[1 * stride + o] = out[DISCOEB_SRC_S3].d;
            fd4[2 * stride + o] = out[DISCOEB_SRC_S4].d;
            fd4[3 * stride + o] = out[DISCOEB_SRC_POTENTIAL].d;
            if (se_dot) se_dot[o] = out[DISCOEB_SRC_E].d;  // the E-mode source has no spline part
        }
        tm.sync();  // the next direction overwrites ypd
    }
}

__device__ Dual spline_slope_dual(Dual x0, Dual x1, Dual y0, Dual y1, Dual S0, Dual S1, Dual xn)
{
    const Dual h = x1 - x0, dx = xn - x0;
    const Dual b = (y1 - y0) / h - h * (S1 + 2.0 * S0) / 6.0, c = S0 / 2.0, dd = (S1 - S0) / (6.0 * h);
    return b + 2.0 * c * dx + 3.0 * dd * dx * dx;
}

// isw_kernel in dual numbers, a block per (direction, mode): the spline of the potential along
// tau with moving knots, its slope at the knots, times exp(-optical depth); S_dot = S1' + S2' +
// S3' + S4'.  pot: the base point's potential rows [n_modes, n_tau]; scratch 4 n_dir n_modes n_tau
__global__ void __launch_bounds__(64) isw_dot_kernel(int n_dir, int n_modes, int n_tau, const double* __restrict__ tau,
                               const double* __restrict__ tau_dot, const double* __restrict__ bt,
                               const double* __restrict__ bt_dot, const double* __restrict__ pot,
                               const double* __restrict__ fd4, double* scratch, double* S_dot)
{
    const int t = blockIdx.x;
    const int d = t / n_modes, im = t - d * n_modes;
    const size_t np = (size_t)n_modes * n_tau, stride = (size_t)n_dir * np;
    const size_t row = (size_t)im * n_tau, drow = (size_t)d * np + row;
    const double* pv = pot + row;
    const double* pd = fd4 + 3 * stride + drow;
    const double* td = tau_dot + (size_t)d * n_tau;
    double* Sv = scratch + drow;
    double* Sd = scratch + stride + drow;
    double* cpv = scratch + 2 * stride + drow;
    double* cpd = scratch + 3 * stride + drow;
    if (threadIdx.x == 0) spline_second_dual(n_tau, tau, td, pv, pd, 1, Sv, Sd, cpv, cpd);
    __syncthreads();
    for (int j = threadIdx.x; j < n_tau; j += blockDim.x) {
        const int i = spline_interval(tau, 1, n_tau, tau[j]);
        const Dual slope = spline_slope_dual(Dual(tau[i], td[i]), Dual(tau[i + 1], td[i + 1]), Dual(pv[i], pd[i]),
                                             Dual(pv[i + 1], pd[i + 1]), Dual(Sv[i], Sd[i]),
                                             Dual(Sv[i + 1], Sd[i + 1]), Dual(tau[j], td[j]));
        const Dual od(bt[DISCOEB_BG_OPTICAL_DEPTH * n_tau + j],
                      bt_dot[((size_t)d * DISCOEB_BG_NFIELDS + DISCOEB_BG_OPTICAL_DEPTH) * n_tau + j]);
        const Dual s1 = xexp(-od) * slope;
        const size_t o = drow + j;
        S_dot[o] = s1.d + fd4[o] + fd4[stride + o] + fd4[2 * stride + o];
    }
}

// ------------------------------------------------------------------------------------------
// workspace layout of discoeb_los (byte offsets, 256-byte aligned)

// how the frequency sum is contracted: DISCOEB_LOS_FP64 (cuBLAS DGEMM) or DISCOEB_LOS_INT8
// (discoeb_dgemm_i8 with `slices` digit planes); library-wide, read once per call
struct LosContraction {
    int kind, slices;
};
std::atomic<int> g_los_kind{DISCOEB_LOS_INT8};
std::atomic<int> g_los_slices{7};

LosContraction los_contraction() { return {g_los_kind.load(), g_los_slices.load()}; }

struct LosLayout {
    size_t sd, s2k, lk, cpk, kd, s2c, cpc, lchi, fidx, fx, fbias, geom, fft, B, cufft, cublas, i8, total;
    long long pitch;
    int n_rows, n_freq;
    LosContraction con;
};

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

constexpr size_t kCublasWorkspace = 32u << 20;

LosLayout los_layout(int n_modes, int n_tau, int ellmax, int n_fft, int n_dense, size_t cufft_bytes,
                     LosContraction con)
{
    LosLayout L;
    L.con = con;
    L.n_rows = n_dense > 0 ? n_dense : n_modes;
    L.n_freq = n_fft / 2 + 1;
    L.pitch = 2LL * L.n_freq;
    size_t o = 0;
    auto take = [&](size_t bytes) { const size_t at = o; o = align256(o + bytes); return at; };
    L.sd = take(n_dense > 0 ? sizeof(double) * (size_t)n_dense * n_tau : 0);
    L.s2k = take(n_dense > 0 ? sizeof(double) * (size_t)n_modes * n_tau : 0);
    L.lk = take(sizeof(double) * (size_t)n_modes);
    L.cpk = take(n_dense > 0 ? sizeof(double) * (size_t)n_modes * n_tau : 0);
    L.kd = take(sizeof(double) * (size_t)L.n_rows);
    L.s2c = take(sizeof(double) * (size_t)L.n_rows * n_tau);
    L.cpc = take(sizeof(double) * (size_t)L.n_rows * n_tau);
    L.lchi = take(sizeof(double) * (size_t)n_tau);
    L.fidx = take(sizeof(int) * (size_t)n_fft);
    L.fx = take(sizeof(double) * (size_t)n_fft);
    L.fbias = take(sizeof(double) * (size_t)n_fft);
    L.geom = take(sizeof(double) * 2);
    L.fft = take(sizeof(double) * (size_t)L.n_rows * L.pitch);
    L.B = take(sizeof(double) * (size_t)(ellmax + 1) * L.pitch);
    L.cufft = take(cufft_bytes);
    L.cublas = take(kCublasWorkspace);
    const int64_t i8 = con.kind == DISCOEB_LOS_INT8
                           ? dgemm_i8::workspace_bytes(L.n_rows, ellmax + 1, (int)L.pitch, con.slices, 0)
                           : 0;
    L.i8 = take(i8 > 0 ? (size_t)i8 : 0);
    L.total = o;
    return L;
}

std::mutex g_blas_mu;
cublasHandle_t g_blas[64] = {};

cublasHandle_t blas_handle(int dev)
{
    if (dev < 0 || dev >= 64) return nullptr;
    if (!g_blas[dev] && cublasCreate(&g_blas[dev]) != CUBLAS_STATUS_SUCCESS) g_blas[dev] = nullptr;
    return g_blas[dev];
}

inline unsigned blocks_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// grid of the row kernels: columns in x (coalesced); in y as many row groups as fill the device a few
// times over (each thread forms its column's constants once for all its rows)
inline dim3 row_grid(int n_rows, int n_cols, int threads)
{
    const unsigned x = blocks_for(n_cols, threads);
    return dim3(x, std::max(1u, std::min((unsigned)n_rows, 4096u / x)));
}

// Scratch of discoeb_sources_noalloc, for callers that cannot allocate device memory: one
// file-scope device array (8 MiB) that every GPU loading the library holds until exit, so the
// call itself allocates nothing.  It holds the per-mode spline recurrence of the ISW term, which
// is written before it is read, so nothing has to be cleared between calls; calls overlapping on
// the GPU share it and race.  Host code must not pass the symbol itself to a kernel (on the host
// it names a stand-in, not device memory): noalloc_scratch() looks up the device address.
constexpr long long kNoAllocScratchDoubles = 1LL << 20;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {};

// device address of g_noalloc_scratch on the current device, looked up once per device (on the
// first no-allocation call made with that device current) and kept for the life of the process:
// a device reset (cudaDeviceReset) unloads the module, after which the kept address is stale, so
// the no-allocation entry is not for processes that reset a device they have used it on
double* noalloc_scratch(int dev)
{
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
            cudaGetLastError();  // clear the error: it belongs to this call, not to the next one
            return nullptr;
        }
        g_noalloc_ptr[dev] = static_cast<double*>(p);
    }
    return g_noalloc_ptr[dev];
}

// Steps 1-5 of the line of sight (the body of discoeb_los) for validated arguments: workspace
// `ws` (256-byte aligned) carved by los_layout, theta [rows, ellmax + 1] written by the GEMM.
// Intermediates stay in the workspace: the dense rows, ln chi knots, FFTLog points, the
// coefficient rows c_q k^-(p_q+1) (`fft`) and the table M_l(p_q) (`B`).
int32_t los_forward(int32_t n_modes, const double* kmodes, int32_t n_tau, const double* tau, const double* S,
                    double tau0, int32_t ellmax, int32_t n_fftlog, int32_t n_k_dense, char* ws, int64_t workspace_bytes,
                    double* theta, double* kmodes_out, void* stream)
{
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int rows = n_k_dense > 0 ? n_k_dense : n_modes;
    const long long pitch = 2LL * (n_fftlog / 2 + 1);
    cufftHandle plan;
    size_t work = 0;
    std::unique_lock<std::mutex> fft_lock(discoeb_fft::plan_mutex());
    if (!discoeb_fft::cached_plan(CUFFT_D2Z, n_fftlog, rows, pitch, pitch / 2, &plan, &work)) return DISCOEB_ECUDA;
    const LosLayout L = los_layout(n_modes, n_tau, ellmax, n_fftlog, n_k_dense, work, los_contraction());
    if ((uint64_t)workspace_bytes < L.total) return DISCOEB_EINVAL;
    auto D = [&](size_t off) { return reinterpret_cast<double*>(ws + off); };
    const int T = 256;
    // 1. rows of S on the k grid used for the integral
    const double* Srow = S;
    const double* krow = kmodes;
    log_kernel<<<blocks_for(n_modes, T), T, 0, s>>>(n_modes, kmodes, D(L.lk));
    if (n_k_dense > 0) {
        k_spline_log_kernel<<<blocks_for(n_tau, 64), 64, 0, s>>>(n_modes, D(L.lk), n_tau, S, D(L.s2k), D(L.cpk));
        k_dense_kernel<<<blocks_for((long long)n_k_dense * n_tau, T), T, 0, s>>>(n_modes, D(L.lk), n_tau, S, D(L.s2k),
                                                                                  n_k_dense, D(L.sd), D(L.kd));
        Srow = D(L.sd);
        krow = D(L.kd);
    } else {
        cudaMemcpyAsync(D(L.kd), kmodes, sizeof(double) * n_modes, cudaMemcpyDeviceToDevice, s);
        krow = D(L.kd);
    }
    cudaMemcpyAsync(kmodes_out, krow, sizeof(double) * rows, cudaMemcpyDeviceToDevice, s);
    // 2. the FFTLog grid and the biased source on it
    geom_kernel<<<1, 32, 0, s>>>(n_tau, tau, tau0, n_fftlog, D(L.geom));
    lchi_kernel<<<blocks_for(n_tau, T), T, 0, s>>>(n_tau, tau, tau0, D(L.lchi));
    fgrid_kernel<<<blocks_for(n_fftlog, T), T, 0, s>>>(n_tau, D(L.lchi), n_fftlog, D(L.geom),
                                                       reinterpret_cast<int*>(ws + L.fidx), D(L.fx), D(L.fbias));
    chi_spline_kernel<<<blocks_for(rows, 64), 64, 0, s>>>(rows, n_tau, D(L.lchi), Srow, D(L.s2c), D(L.cpc));
    chi_eval_kernel<<<row_grid(rows, n_fftlog, T), T, 0, s>>>(
        rows, n_tau, D(L.lchi), Srow, D(L.s2c), n_fftlog, reinterpret_cast<const int*>(ws + L.fidx), D(L.fx),
        D(L.fbias), L.pitch, D(L.fft));
    // 3. rfft of every row, in place (the plan lock is held from the lookup to here, so no other
    //    call can evict the plan or change its work area in between)
    cufftSetWorkArea(plan, ws + L.cufft);
    cufftSetStream(plan, s);
    const cufftResult fr = cufftExecD2Z(plan, D(L.fft), reinterpret_cast<cufftDoubleComplex*>(D(L.fft)));
    fft_lock.unlock();
    if (fr != CUFFT_SUCCESS) return DISCOEB_ECUDA;
    // 4. ck in place, and the M table
    ck_kernel<<<rows, kPhaseThreads, 0, s>>>(rows, krow, n_fftlog, L.n_freq, D(L.geom),
                                                                      L.pitch, D(L.fft));
    mcoef_kernel<<<blocks_for(mcoef_threads(ellmax + 1, L.n_freq), T), T, 0, s>>>(ellmax + 1, L.n_freq, n_fftlog,
                                                                                 D(L.geom), nullptr, D(L.B), nullptr);
    if (cudaGetLastError() != cudaSuccess) return DISCOEB_ECUDA;
    // 5. theta[r, l] = sum_j A[r, j] B[l, j] over the interleaved (re, im) pairs: one product,
    //    on the int8 tensor cores (digit planes, exact int32 sums) or as a cuBLAS DGEMM
    if (L.con.kind == DISCOEB_LOS_INT8)
        return dgemm_i8::run(rows, ellmax + 1, (int)L.pitch, D(L.fft), L.pitch, false, D(L.B), L.pitch, false, theta,
                             ellmax + 1, L.con.slices, 0, ws + L.i8, (int64_t)(L.total - L.i8), stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    std::lock_guard<std::mutex> lock(g_blas_mu);
    cublasHandle_t h = blas_handle(dev);
    if (!h) return DISCOEB_ECUDA;
    cublasSetStream(h, s);
    cublasSetWorkspace(h, ws + L.cublas, kCublasWorkspace);
    const double one = 1.0, zero = 0.0;
    const cublasStatus_t st =
        cublasDgemm(h, CUBLAS_OP_T, CUBLAS_OP_N, ellmax + 1, rows, (int)L.pitch, &one, D(L.B), (int)L.pitch, D(L.fft),
                    (int)L.pitch, &zero, theta, ellmax + 1);
    cublasSetWorkspace(h, nullptr, 0);
    if (st != CUBLAS_STATUS_SUCCESS) return DISCOEB_ECUDA;
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}


// workspace of discoeb_los_cell_jvp: the line of sight's own (los_layout) followed by these
struct LosJvpLayout {
    LosLayout base;
    size_t th, G, H, Bd, Fd, w, kout, kscratch, sdd, s2kd, cpkd, lchid, fxd, fbd, gd, S2v, S2d, cpv, cpd, i8t, total;
};

LosJvpLayout los_jvp_layout(int n_modes, int n_tau, int ellmax, int n_fft, int n_dense, size_t cufft_bytes)
{
    LosJvpLayout J;
    J.base = los_layout(n_modes, n_tau, ellmax, n_fft, n_dense, cufft_bytes, los_contraction());
    const size_t rows = (size_t)J.base.n_rows, L = (size_t)ellmax + 1, pitch = (size_t)J.base.pitch;
    size_t o = J.base.total;
    auto take = [&](size_t doubles) { const size_t at = o; o = align256(o + sizeof(double) * doubles); return at; };
    J.th = take(rows * L);
    J.G = take(L * pitch);
    J.H = take(L * pitch);
    J.Bd = take(L * pitch);
    J.Fd = take(rows * pitch);
    J.w = take(rows);
    J.kout = take(rows);
    J.kscratch = take(rows);
    J.sdd = take(n_dense > 0 ? (size_t)n_dense * n_tau : 0);
    J.s2kd = take(n_dense > 0 ? (size_t)n_modes * n_tau : 0);
    J.cpkd = take(n_dense > 0 ? (size_t)n_modes * n_tau : 0);
    J.lchid = take(n_tau);
    J.fxd = take(n_fft);
    J.fbd = take(n_fft);
    J.gd = take(2);
    J.S2v = take(rows * n_tau);
    J.S2d = take(rows * n_tau);
    J.cpv = take(rows * n_tau);
    J.cpd = take(rows * n_tau);
    // the int8 form of Omega^T A ([L, pitch] over the modes): its own digit planes and level sums
    const int64_t i8t = J.base.con.kind == DISCOEB_LOS_INT8
                            ? dgemm_i8::workspace_bytes((int)L, (int)pitch, (int)rows, J.base.con.slices, 0)
                            : 0;
    J.i8t = take(i8t > 0 ? (size_t)i8t / sizeof(double) + 1 : 0);
    J.total = o;
    return J;
}

bool los_args_ok(int n_modes, int n_tau, int ellmax, int n_fftlog, int n_k_dense)
{
    return !(n_modes < 2 || n_tau < 3 || ellmax < 0 || n_fftlog < 2 || n_k_dense < 0 || n_k_dense == 1);
}

// cuFFT work-area size of the line of sight's batched transform (plan made and cached)
bool los_fft_work(int n_fftlog, int rows, size_t* work)
{
    const long long pitch = 2LL * (n_fftlog / 2 + 1);
    cufftHandle plan;
    std::lock_guard<std::mutex> lock(discoeb_fft::plan_mutex());
    return discoeb_fft::cached_plan(CUFFT_D2Z, n_fftlog, rows, pitch, pitch / 2, &plan, work);
}

}  // namespace

extern "C" {

int32_t discoeb_sources(const DiscoebCosmo* cosmo_dev, const DiscoebCosmo* cosmo_host, int32_t n_modes,
                        const double* kmodes, int32_t n_tau, const double* tau, const double* bgtab,
                        const double* y_full, double* fields, double* scratch, void* stream)
{
    if (!cosmo_host || !cosmo_dev || n_modes < 0 || n_tau < 0) return DISCOEB_EINVAL;
    if (cosmo_host->use_tca) return DISCOEB_EUNSUPPORTED;
    if (n_modes == 0 || n_tau == 0) return DISCOEB_SUCCESS;
    if (n_tau < 3 || !kmodes || !tau || !bgtab || !y_full || !fields || !scratch) return DISCOEB_EINVAL;
    const Dims D = make_dims(*cosmo_host);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const long long points = (long long)n_modes * n_tau;
    const int threads = 128;
    if (points * 32 / threads >= 0x7fffffffLL) return DISCOEB_EINVAL;  // one warp per point must fit the grid
    const size_t smem = sizeof(double) * (size_t)D.n * (threads / 32);
    sources_kernel<<<blocks_for(points * 32, threads), threads, smem, s>>>(cosmo_dev, n_modes, kmodes, n_tau, tau,
                                                                            bgtab, y_full, fields);
    isw_kernel<<<n_modes, 64, 0, s>>>(n_modes, n_tau, tau, bgtab, fields, scratch);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int32_t discoeb_fwd_sources(const DiscoebCosmo* cosmo_dev, const DiscoebCosmo* cosmo_host,
                            const DiscoebControl* ctrl, int32_t n_modes, const double* kmodes, const double* tau_start,
                            const double* y0, const double* switch_tau, int32_t n_tau, const double* tau,
                            const double* bgtab, double* y_full, double* fields, double* scratch, int32_t* status,
                            int32_t* nsteps, void* stream)
{
    if (!cosmo_host || !cosmo_dev || !ctrl || n_modes < 0 || n_tau < 0) return DISCOEB_EINVAL;
    if (cosmo_host->use_tca) return DISCOEB_EUNSUPPORTED;
    if (cosmo_host->nqmax < 0 || cosmo_host->nqmax > DISCOEB_MAX_NQ) return DISCOEB_EINVAL;
    if (ctrl->method != DISCOEB_METHOD_RODAS5_STRUCTURED) return DISCOEB_EUNSUPPORTED;
    if (!(ctrl->rtol > 0.0) || !(ctrl->atol >= 0.0) || ctrl->max_steps < 1) return DISCOEB_EINVAL;
    if (n_modes == 0 || n_tau == 0) return DISCOEB_SUCCESS;
    if (n_tau < 3 || !kmodes || !tau_start || !y0 || !switch_tau || !tau || !bgtab || !fields || !scratch ||
        !status || !nsteps)
        return DISCOEB_EINVAL;
    if ((long long)n_modes * n_tau > 0x7fffffffLL) return DISCOEB_EINVAL;
    const Dims D = make_dims(*cosmo_host);
    const int mem = mode_mem_doubles(D);
    const size_t smem = (size_t)(kCosmoDoublesC + mem) * sizeof(double);
    int dev = 0, max_optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem > (size_t)max_optin) return DISCOEB_EUNSUPPORTED;
    if (cudaFuncSetAttribute(fwd_sources_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DISCOEB_ECUDA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    fwd_sources_kernel<<<n_modes, 32, smem, s>>>(cosmo_dev, *ctrl, n_modes, kmodes, tau_start, y0, switch_tau, n_tau,
                                                  tau, bgtab, mem, y_full, fields, status, nsteps);
    isw_kernel<<<n_modes, 64, 0, s>>>(n_modes, n_tau, tau, bgtab, fields, scratch);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int32_t discoeb_sources_noalloc(const DiscoebCosmo* cosmo_dev, const DiscoebCosmo* cosmo_host, int32_t n_modes,
                                const double* kmodes, int32_t n_tau, const double* tau, const double* bgtab,
                                const double* y_full, double* fields, void* stream)
{
    if (n_modes < 0 || n_tau < 0) return DISCOEB_EINVAL;
    if ((long long)n_modes * n_tau > kNoAllocScratchDoubles) return DISCOEB_EINVAL;
    if (n_modes == 0 || n_tau == 0) return discoeb_sources(cosmo_dev, cosmo_host, n_modes, kmodes, n_tau, tau, bgtab,
                                                           y_full, fields, nullptr, stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    double* scratch = noalloc_scratch(dev);
    if (!scratch) return DISCOEB_ECUDA;
    return discoeb_sources(cosmo_dev, cosmo_host, n_modes, kmodes, n_tau, tau, bgtab, y_full, fields, scratch, stream);
}

int64_t discoeb_los_workspace_bytes(int32_t n_modes, int32_t n_tau, int32_t ellmax, int32_t n_fftlog,
                                    int32_t n_k_dense)
{
    if (n_modes < 2 || n_tau < 3 || ellmax < 0 || n_fftlog < 2 || n_k_dense < 0 || n_k_dense == 1)
        return DISCOEB_EINVAL;
    const int rows = n_k_dense > 0 ? n_k_dense : n_modes;
    const long long pitch = 2LL * (n_fftlog / 2 + 1);
    cufftHandle plan;
    size_t work = 0;
    std::lock_guard<std::mutex> lock(discoeb_fft::plan_mutex());
    if (!discoeb_fft::cached_plan(CUFFT_D2Z, n_fftlog, rows, pitch, pitch / 2, &plan, &work)) return DISCOEB_ECUDA;
    return (int64_t)los_layout(n_modes, n_tau, ellmax, n_fftlog, n_k_dense, work, los_contraction()).total;
}

int32_t discoeb_set_los_contraction(int32_t kind, int32_t slices)
{
    if (kind != DISCOEB_LOS_FP64 && kind != DISCOEB_LOS_INT8) return DISCOEB_EINVAL;
    if (kind == DISCOEB_LOS_INT8 && (slices < 1 || slices > dgemm_i8::kMaxSlices)) return DISCOEB_EINVAL;
    g_los_slices.store(kind == DISCOEB_LOS_INT8 ? slices : g_los_slices.load());
    g_los_kind.store(kind);
    return DISCOEB_SUCCESS;
}

int32_t discoeb_get_los_contraction(int32_t* kind, int32_t* slices)
{
    if (!kind || !slices) return DISCOEB_EINVAL;
    *kind = g_los_kind.load();
    *slices = g_los_slices.load();
    return DISCOEB_SUCCESS;
}

int32_t discoeb_los(int32_t n_modes, const double* kmodes, int32_t n_tau, const double* tau, const double* S,
                    double tau0, int32_t ellmax, int32_t n_fftlog, int32_t n_k_dense, void* workspace,
                    int64_t workspace_bytes, double* theta, double* kmodes_out, void* stream)
{
    if (n_modes < 2 || n_tau < 3 || ellmax < 0 || n_fftlog < 2 || n_k_dense < 0 || n_k_dense == 1)
        return DISCOEB_EINVAL;
    if (!kmodes || !tau || !S || !workspace || !theta || !kmodes_out) return DISCOEB_EINVAL;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return DISCOEB_EINVAL;
    return los_forward(n_modes, kmodes, n_tau, tau, S, tau0, ellmax, n_fftlog, n_k_dense,
                       static_cast<char*>(workspace), workspace_bytes, theta, kmodes_out, stream);
}

int32_t discoeb_cell(int32_t n_modes, const double* kmodes, int32_t n_ell, const double* theta, double n_s, double k_p,
                     double* cell, void* stream)
{
    if (n_modes < 2 || n_ell < 1 || !kmodes || !theta || !cell) return DISCOEB_EINVAL;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cell_kernel<<<(n_ell + 31) / 32, 256, 0, s>>>(n_modes, kmodes, n_ell, theta, n_s, k_p, cell);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int32_t discoeb_cell_cross(int32_t n_modes, const double* kmodes, int32_t n_ell, const double* theta_a,
                           const double* theta_b, double n_s, double k_p, double* cell, void* stream)
{
    if (n_modes < 2 || n_ell < 1 || !kmodes || !theta_a || !theta_b || !cell) return DISCOEB_EINVAL;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cell_kernel<<<(n_ell + 31) / 32, 256, 0, s>>>(n_modes, kmodes, n_ell, theta_a, n_s, k_p, cell, false, theta_b);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

static int64_t e_align(int64_t b) { return (b + 255) / 256 * 256; }

int64_t discoeb_los_e_workspace_bytes(int32_t n_modes, int32_t n_tau, int32_t ellmax, int32_t n_fftlog,
                                      int32_t n_k_dense)
{
    if (ellmax < 0 || ellmax > 0x7ffffff0) return DISCOEB_EINVAL;
    const int64_t b = discoeb_los_workspace_bytes(n_modes, n_tau, ellmax + 2, n_fftlog, n_k_dense);
    if (b < 0) return b;
    const int64_t rows = n_k_dense > 0 ? n_k_dense : n_modes;
    return e_align((int64_t)n_modes * n_tau * 8) + e_align(rows * (ellmax + 3) * 8) + b;
}

int32_t discoeb_los_e(int32_t n_modes, const double* kmodes, int32_t n_tau, const double* tau, const double* S_E,
                      double tau0, int32_t ellmax, int32_t n_fftlog, int32_t n_k_dense, void* workspace,
                      int64_t workspace_bytes, double* theta, double* kmodes_out, void* stream)
{
    if (n_modes < 2 || n_tau < 3 || ellmax < 0 || n_fftlog < 2 || n_k_dense < 0 || n_k_dense == 1)
        return DISCOEB_EINVAL;
    if (!kmodes || !tau || !S_E || !workspace || !theta || !kmodes_out) return DISCOEB_EINVAL;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return DISCOEB_EINVAL;
    const int64_t need = discoeb_los_e_workspace_bytes(n_modes, n_tau, ellmax, n_fftlog, n_k_dense);
    if (need < 0) return (int32_t)need;
    if (workspace_bytes < need) return DISCOEB_EINVAL;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int rows = n_k_dense > 0 ? n_k_dense : n_modes;
    const int n_ell = ellmax + 1, nlo = n_ell < kELSwitch ? n_ell : kELSwitch;
    char* ws = static_cast<char*>(workspace);
    double* Sx = reinterpret_cast<double*>(ws);
    const int64_t o1 = e_align((int64_t)n_modes * n_tau * 8);
    double* th = reinterpret_cast<double*>(ws + o1);
    const int64_t o2 = o1 + e_align((int64_t)rows * (ellmax + 3) * 8);
    const long long pts = (long long)n_modes * n_tau;
    // l < nlo: S_E / chi^2
    e_source_kernel<<<blocks_for(pts, 256), 256, 0, s>>>(n_modes, n_tau, tau, tau0, S_E, Sx);
    int32_t rc = los_forward(n_modes, kmodes, n_tau, tau, Sx, tau0, nlo - 1, n_fftlog, n_k_dense, ws + o2,
                             workspace_bytes - o2, th, kmodes_out, stream);
    if (rc != DISCOEB_SUCCESS) return rc;
    e_low_kernel<<<blocks_for((long long)rows * nlo, 256), 256, 0, s>>>(rows, n_ell, nlo, kmodes_out, th, theta);
    if (n_ell > nlo) {  // l >= nlo: S_E at l - 2, l, l + 2
        rc = los_forward(n_modes, kmodes, n_tau, tau, S_E, tau0, ellmax + 2, n_fftlog, n_k_dense, ws + o2,
                         workspace_bytes - o2, th, kmodes_out, stream);
        if (rc != DISCOEB_SUCCESS) return rc;
        e_high_kernel<<<blocks_for((long long)rows * (n_ell - nlo), 256), 256, 0, s>>>(rows, n_ell, nlo, th, theta);
    }
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int64_t discoeb_los_cell_jvp_workspace_bytes(int32_t n_modes, int32_t n_tau, int32_t ellmax, int32_t n_fftlog,
                                             int32_t n_k_dense)
{
    if (!los_args_ok(n_modes, n_tau, ellmax, n_fftlog, n_k_dense)) return DISCOEB_EINVAL;
    size_t work = 0;
    if (!los_fft_work(n_fftlog, n_k_dense > 0 ? n_k_dense : n_modes, &work)) return DISCOEB_ECUDA;
    return (int64_t)los_jvp_layout(n_modes, n_tau, ellmax, n_fftlog, n_k_dense, work).total;
}

int32_t discoeb_los_cell_jvp(int32_t n_modes, const double* kmodes, int32_t n_tau, const double* tau, const double* S,
                             double tau0, int32_t n_dir, const double* tau_dot, const double* S_dot,
                             const double* tau0_dot, int32_t ellmax, int32_t n_fftlog, int32_t n_k_dense, double n_s,
                             double k_p, void* workspace, int64_t workspace_bytes, double* cell, double* cell_dot,
                             double* cell_dns, void* stream)
{
    if (!los_args_ok(n_modes, n_tau, ellmax, n_fftlog, n_k_dense) || n_dir < 0) return DISCOEB_EINVAL;
    if (!kmodes || !tau || !S || !workspace || !cell) return DISCOEB_EINVAL;
    if (n_dir > 0 && (!tau_dot || !S_dot || !tau0_dot || !cell_dot)) return DISCOEB_EINVAL;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return DISCOEB_EINVAL;
    const int rows = n_k_dense > 0 ? n_k_dense : n_modes;
    size_t work = 0;
    if (!los_fft_work(n_fftlog, rows, &work)) return DISCOEB_ECUDA;
    const LosJvpLayout J = los_jvp_layout(n_modes, n_tau, ellmax, n_fftlog, n_k_dense, work);
    if ((uint64_t)workspace_bytes < J.total) return DISCOEB_EINVAL;
    const LosLayout& L = J.base;
    char* ws = static_cast<char*>(workspace);
    auto D = [&](size_t off) { return reinterpret_cast<double*>(ws + off); };
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int n_ell = ellmax + 1, T = 256;
    const long long pitch = L.pitch;
    // base point: Theta, C_l, Omega = w Theta (in place), G = Omega^T A
    int rc = los_forward(n_modes, kmodes, n_tau, tau, S, tau0, ellmax, n_fftlog, n_k_dense, ws, (int64_t)L.total,
                         D(J.th), D(J.kout), stream);
    if (rc) return rc;
    cell_kernel<<<(n_ell + 31) / 32, 256, 0, s>>>(rows, D(J.kout), n_ell, D(J.th), n_s, k_p, cell);
    if (cell_dns) cell_kernel<<<(n_ell + 31) / 32, 256, 0, s>>>(rows, D(J.kout), n_ell, D(J.th), n_s, k_p, cell_dns, true);
    if (n_dir == 0) return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
    cell_weight_kernel<<<blocks_for(rows, T), T, 0, s>>>(rows, D(J.kout), n_s, k_p, D(J.w));
    scale_rows_kernel<<<blocks_for((long long)rows * n_ell, T), T, 0, s>>>(rows, n_ell, D(J.w), D(J.th));
    if (cudaGetLastError() != cudaSuccess) return DISCOEB_ECUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DISCOEB_ECUDA;
    const double one = 1.0, zero = 0.0;
    auto omega_t_times = [&](const double* A, double* out) {  // out [n_ell, pitch] = Omega^T A
        if (L.con.kind == DISCOEB_LOS_INT8)  // both operands K-major over the modes
            return dgemm_i8::run(n_ell, (int)pitch, rows, D(J.th), n_ell, true, A, pitch, true, out, pitch,
                                 L.con.slices, 0, ws + J.i8t, (int64_t)(J.total - J.i8t), stream) == DISCOEB_SUCCESS;
        std::lock_guard<std::mutex> lock(g_blas_mu);
        cublasHandle_t h = blas_handle(dev);
        if (!h) return false;
        cublasSetStream(h, s);
        cublasSetWorkspace(h, ws + L.cublas, kCublasWorkspace);
        const cublasStatus_t st = cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, (int)pitch, n_ell, rows, &one, A, (int)pitch,
                                              D(J.th), n_ell, &zero, out, (int)pitch);
        cublasSetWorkspace(h, nullptr, 0);
        return st == CUBLAS_STATUS_SUCCESS;
    };
    if (!omega_t_times(D(L.fft), D(J.G))) return DISCOEB_ECUDA;
    const double* Srow = n_k_dense > 0 ? D(L.sd) : S;
    for (int d = 0; d < n_dir; ++d) {
        const double* Sd_in = S_dot + (size_t)d * n_modes * n_tau;
        const double* td = tau_dot + (size_t)d * n_tau;
        const double* Srow_dot = Sd_in;
        if (n_k_dense > 0) {  // the dense-k resampling is linear in S and k is fixed
            k_spline_log_kernel<<<blocks_for(n_tau, 64), 64, 0, s>>>(n_modes, D(L.lk), n_tau, Sd_in, D(J.s2kd),
                                                                      D(J.cpkd));
            k_dense_kernel<<<blocks_for((long long)n_k_dense * n_tau, T), T, 0, s>>>(
                n_modes, D(L.lk), n_tau, Sd_in, D(J.s2kd), n_k_dense, D(J.sdd), D(J.kscratch));
            Srow_dot = D(J.sdd);
        }
        geom_dot_kernel<<<1, 32, 0, s>>>(n_tau, tau, td, tau0, tau0_dot[d], n_fftlog, D(J.gd));
        lchi_dot_kernel<<<blocks_for(n_tau, T), T, 0, s>>>(n_tau, tau, td, tau0, tau0_dot[d], D(J.lchid));
        fgrid_dot_kernel<<<blocks_for(n_fftlog, T), T, 0, s>>>(n_fftlog, D(J.gd), D(L.fbias), D(J.fxd), D(J.fbd));
        chi_spline_dot_kernel<<<blocks_for(rows, 64), 64, 0, s>>>(rows, n_tau, D(L.lchi), D(J.lchid), Srow, Srow_dot,
                                                                  D(J.S2v), D(J.S2d), D(J.cpv), D(J.cpd));
        chi_eval_dot_kernel<<<row_grid(rows, n_fftlog, T), T, 0, s>>>(
            rows, n_tau, D(L.lchi), D(J.lchid), Srow, Srow_dot, D(J.S2v), D(J.S2d), n_fftlog,
            reinterpret_cast<const int*>(ws + L.fidx), D(L.fx), D(J.fxd), D(L.fbias), D(J.fbd), pitch, D(J.Fd));
        {
            cufftHandle plan;
            size_t w2 = 0;
            std::lock_guard<std::mutex> lock(discoeb_fft::plan_mutex());
            if (!discoeb_fft::cached_plan(CUFFT_D2Z, n_fftlog, rows, pitch, pitch / 2, &plan, &w2) || w2 > work)
                return DISCOEB_ECUDA;
            cufftSetWorkArea(plan, ws + L.cufft);
            cufftSetStream(plan, s);
            if (cufftExecD2Z(plan, D(J.Fd), reinterpret_cast<cufftDoubleComplex*>(D(J.Fd))) != CUFFT_SUCCESS)
                return DISCOEB_ECUDA;
        }
        ck_dot_kernel<<<rows, kPhaseThreads, 0, s>>>(rows, D(L.kd), n_fftlog, L.n_freq,
                                                                              D(L.geom), D(J.gd), pitch, D(L.fft),
                                                                              D(J.Fd));
        mcoef_kernel<<<blocks_for(mcoef_threads(n_ell, L.n_freq), T), T, 0, s>>>(n_ell, L.n_freq, n_fftlog, D(L.geom),
                                                                                 D(J.gd), nullptr, D(J.Bd));
        if (cudaGetLastError() != cudaSuccess) return DISCOEB_ECUDA;
        if (!omega_t_times(D(J.Fd), D(J.H))) return DISCOEB_ECUDA;
        cell_dot_kernel<<<n_ell, 256, 0, s>>>(n_ell, pitch, D(L.B), D(J.H), D(J.Bd), D(J.G), cell_dot + (size_t)d * n_ell);
    }
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

int32_t discoeb_sources_jvp(const DiscoebCosmo* cosmo_dev, const DiscoebCosmo* cosmo_host,
                            const DiscoebTangent* tangents_dev, int32_t n_dir, int32_t n_modes, const double* kmodes,
                            int32_t n_tau, const double* tau, const double* tau_dot, const double* bgtab,
                            const double* bgtab_dot, const double* y_full, const double* y_full_dot,
                            const double* fields, double* S_dot, double* scratch, double* SE_dot, void* stream)
{
    if (!cosmo_host || !cosmo_dev || !tangents_dev || n_dir < 1 || n_modes < 0 || n_tau < 0) return DISCOEB_EINVAL;
    if (cosmo_host->use_tca) return DISCOEB_EUNSUPPORTED;
    if (n_modes == 0 || n_tau == 0) return DISCOEB_SUCCESS;
    if (n_tau < 3 || !kmodes || !tau || !tau_dot || !bgtab || !bgtab_dot || !y_full || !y_full_dot || !fields ||
        !S_dot || !scratch)
        return DISCOEB_EINVAL;
    const Dims D = make_dims(*cosmo_host);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const long long points = (long long)n_dir * n_modes * n_tau;
    const long long warps = (long long)n_modes * n_tau;  // one warp per (mode, time), every direction
    const int threads = 128;
    // isw_dot_kernel indexes (direction, mode) pairs with an int, and one warp per point must fit
    // the grid: larger problems are refused rather than truncated
    if ((long long)n_dir * n_modes > 0x7fffffffLL || warps * 32 / threads >= 0x7fffffffLL) return DISCOEB_EINVAL;
    const size_t smem = sizeof(double) * 2 * (size_t)D.n * (threads / 32);
    double* fd4 = scratch;                       // [4, n_dir, n_modes, n_tau]
    double* sp = scratch + 4 * (size_t)points;  // [4, n_dir, n_modes, n_tau]
    sources_dot_kernel<<<blocks_for(warps * 32, threads), threads, smem, s>>>(
        cosmo_dev, tangents_dev, n_dir, n_modes, kmodes, n_tau, tau, tau_dot, bgtab, bgtab_dot, y_full, y_full_dot, fd4,
        SE_dot);
    const size_t stride = (size_t)n_modes * n_tau;
    isw_dot_kernel<<<n_dir * n_modes, 64, 0, s>>>(
        n_dir, n_modes, n_tau, tau, tau_dot, bgtab, bgtab_dot, fields + DISCOEB_SRC_POTENTIAL * stride, fd4, sp, S_dot);
    return cudaGetLastError() == cudaSuccess ? DISCOEB_SUCCESS : DISCOEB_ECUDA;
}

}  // extern "C"
