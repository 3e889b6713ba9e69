// The one-launch time loop of the PolF64 element type (see star7_loop.cuh).
#include "star7_loop.cuh"

namespace scafes {

cudaError_t launch_star7_loop_f64(const Star7Loop& q, cudaStream_t stream) {
    return launch_loop_prec<PolF64>(q, stream);
}

}  // namespace scafes
