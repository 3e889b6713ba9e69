// The one-launch time loop of the PolF32x2 element type (see star7_loop.cuh).
#include "star7_loop.cuh"

namespace scafes {

cudaError_t launch_star7_loop_f32x2(const Star7Loop& q, cudaStream_t stream) {
    return launch_loop_prec<PolF32x2>(q, stream);
}

}  // namespace scafes
