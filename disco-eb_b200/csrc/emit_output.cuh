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

// TM: WarpTeam (FP64) or WarpTeamMixed (FP32 chain factors, mix_doubles more per warp)
}  // namespace dscb
