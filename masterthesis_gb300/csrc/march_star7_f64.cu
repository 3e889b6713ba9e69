// The sweep by plain loads of the PolF64 element type (see star7_march.cuh).
#include "star7_march.cuh"

namespace scafes {

cudaError_t launch_star7_march_f64(const Star7Launch& a, cudaStream_t stream) {
    return launch_march_prec<PolF64>(a, stream);
}

}  // namespace scafes
