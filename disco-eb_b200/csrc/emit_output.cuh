// The output stage of a forward solve: RSA projection and output fields of one state (device only).
#pragma once

#include "stepper.cuh"

namespace dscb {

// write state / projected state / output fields of one output time (team-parallel)
__device__ inline void emit_output(const WarpTeam& tm, const DiscoebCosmo& P, const Dims& D, double k, double tau,
                            const double* y, double* yfull, double* y20, double* scratch20)
{
    const int n = D.n;
    double fld[4];
    const bool rsa = rsa_projection<double>(P, nullptr, D, tau, k, y, nullptr, fld);  // all lanes, identical
    // projected state into scratch (shared) then outputs
    double* yp = scratch20;  // n doubles of shared scratch
    for (int i = tm.lane; i < n; i += 32) {
        double v = y[i];
        if (rsa) {
            const int s = rsa_slot(D, i);
            if (s >= 0) v = fld[s];
            else if (s == -1) v = 0.0;
        }
        yp[i] = v;
        if (yfull) yfull[i] = v;
    }
    tm.sync();
    if (y20 && tm.leader()) {
        double o[20];
        output_vars<double>(P, nullptr, D, k, yp, nullptr, o);
        for (int q = 0; q < 20; ++q) y20[q] = o[q];
    }
    tm.sync();
}

// Output fields and their tangents at output time j of one (mode, direction): the tangent of
// the state at the moving output time is y' + f tau_out', then the RSA projection and the
// output conversion in dual numbers.  y: the forward state at tau_out[j]; pf: n doubles of
// scratch; TT.fd / TT.jk are used as scratch.  Full: the RSA-projected state and its tangent
// (n values per output) are written instead of the 20 output fields.  Kept out of line: it runs
// at output times only, and inlined into the tangent loop it lengthens the hot code the seven
// warps of a block fetch (measured: the gradient kernel 2% slower inlined).
template <bool Full>
static __device__ __noinline__ void emit_tangent_output(const WarpTeam& tm, const DiscoebCosmo& P, const DiscoebTangent* TN, const Dims& D,
                                    double k, int mode, int dir, int n_modes, int n_out, int j, const double* tau_out,
                                    const double* tau_out_dot, const double* y, int regime, const TanMem& TT,
                                    double* pf, double* y_out20, double* y_out20_dot)
{
    const int n = D.n;
    // f at the output time (left limit of the last step's regime), for the moving output time
    int hint = P.xe_loga.n_knots / 2;
    Bg<double> b;
    bg_eval_team(tm, P, y[0], tau_out[j], k, regime, b, hint);
    rhs_team(tm, P, D, b, k, tau_out[j], y, TT.fd, (double*)nullptr);
    tm.sync();
    const double td = tau_out_dot[(size_t)dir * n_out + j];
    for (int i = tm.lane; i < n; i += 32) TT.jk[i] = TT.yd[i] + TT.fd[i] * td;
    tm.sync();
    Dual fld[4];
    const bool rsa = rsa_projection<Dual>(P, TN, D, tau_out[j], k, y, TT.jk, fld);
    for (int i = tm.lane; i < n; i += 32) {
        double v = y[i], vd = TT.jk[i];
        if (rsa) {
            const int sl = rsa_slot(D, i);
            if (sl >= 0) { v = fld[sl].v; vd = fld[sl].d; }
            else if (sl == -1) { v = 0.0; vd = 0.0; }
        }
        if constexpr (Full) {
            const size_t oo = (size_t)mode * n_out + j;
            y_out20_dot[((size_t)dir * n_modes * n_out + oo) * n + i] = vd;
            if (dir == 0 && y_out20) y_out20[oo * n + i] = v;
        } else {
            pf[i] = v;
            TT.fd[i] = vd;
        }
    }
    tm.sync();
    if constexpr (Full) return;
    if (tm.leader()) {
        Dual o[20];
        output_vars<Dual>(P, TN, D, k, pf, TT.fd, o);
        const size_t oo = (size_t)mode * n_out + j;
        for (int q = 0; q < 20; ++q) y_out20_dot[((size_t)dir * n_modes * n_out + oo) * 20 + q] = o[q].d;
        if (dir == 0 && y_out20)
            for (int q = 0; q < 20; ++q) y_out20[oo * 20 + q] = o[q].v;
    }
    tm.sync();
}

}  // namespace dscb
