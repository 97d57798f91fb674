// Launch of the block solver (solve_block.cuh) for discoeb_fwd and discoeb_fwd_record.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "form_choice.cuh"
#include "stepper.cuh"

namespace dscb {
namespace blk {

// dynamic shared memory of one mode's block (~0 where the state has more rows than a block takes)
size_t smem_bytes(const Dims& D);

// the block form against a warp per mode for n_modes modes on a device of that many SMs
FormChoice forward_choice(const Dims& D, int n_modes, int sms);

// where discoeb_fwd_record's steps go: per mode `doubles` from base on, cap end times, then a start
// state every `every` steps
struct StepRecords {
    double* base;
    long long doubles;
    int cap, every;
    int32_t* n_accepted;
};

// the FP64 solve of discoeb_fwd and, with records, of discoeb_fwd_record (arguments checked by the
// caller); a DISCOEB_* status.  gate: FormChoice's; the caller then launches the other form after it.
int32_t launch_fwd(const DiscoebCosmo* cosmos, int n_cosmo, const int32_t* mode_cosmo, const DiscoebControl& ctrl,
                   int n_modes, const double* kmodes, const double* tau_start, const double* y0, const double* sw,
                   int n_out, const double* tau_out, const Dims& D, double* y_full, double* y_out20, int32_t* status,
                   int32_t* nsteps, const StepRecords* records, int sms, int gate, cudaStream_t stream);

}  // namespace blk
}  // namespace dscb
