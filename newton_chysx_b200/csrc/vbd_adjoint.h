// Launchers of the recorded substep and its reverse (compiled in vbd_adjoint.cu).
#pragma once
#include <vector>

#include "vbd_kernels.cuh"

namespace vbd {

struct ColorLists {
  const int* particles;             // particles by color (device)
  const std::vector<int>* offsets;  // [colors + 1]
  const int* color_of;              // [V] color of each particle (device)
};

// One substep that keeps the inertial targets y [V*3] and the positions at the start of every iteration and at the
// end, ck [(iterations + 1), V*3]; writes c.q_out and c.qd_out.
template <typename R>
cudaError_t record_substep(const StepCtx<R>& c, const ColorLists& l, int iterations, R* y, R* ck, cudaStream_t st);

// Its reverse. work: [3 * V*3].
template <typename R>
cudaError_t adjoint_substep(const StepCtx<R>& c, const ColorLists& l, int iterations, const R* y, const R* ck, R* work,
                            const R* aq_out, const R* aqd_out, R* aq_in, R* aqd_in, R* adj_mu, R* adj_lambda,
                            cudaStream_t st);

}  // namespace vbd
