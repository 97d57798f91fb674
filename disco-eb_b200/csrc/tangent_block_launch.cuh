// Launch of the block form of discoeb_jvp (tangent_block.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "form_choice.cuh"
#include "stepper.cuh"

namespace dscb {
namespace blk {

// directions of one block, at most `want` (0: the state is too large for this form), and its shared memory
int jvp_directions(const Dims& D, int want, size_t max_smem, size_t& smem);

// discoeb_jvp (full: discoeb_jvp_full), arguments checked by the caller, nd directions per block.  gate:
// FormChoice's; the caller then launches the older kernel after it
template <bool Full>
int32_t launch_jvp_block(const DiscoebCosmo* cosmos, int n_cosmo, const int32_t* mode_cosmo,
                         const DiscoebTangent* tangents, int n_dir, int nd, size_t smem, const Dims& D,
                         const DiscoebControl& ctrl, int n_modes, const double* kmodes, const double* tau_start,
                         const double* y0, const double* y0_dot, const double* sw, int n_out, const double* tau_out,
                         const double* tau_out_dot, double* y_out, double* y_out_dot, int32_t* status, int32_t* nsteps,
                         int gate, cudaStream_t stream);

}  // namespace blk
}  // namespace dscb
