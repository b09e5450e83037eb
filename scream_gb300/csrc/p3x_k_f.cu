/* Column kernel instantiation: rate type float. */
#include "p3x_kernels_impl.cuh"

namespace p3x {
template cudaError_t launch_p3_part<float>(const dev::Inst&, const dev::KParams<float>&,
                                                 const LaunchSpec&, int, int, cudaStream_t);
}  // namespace p3x
