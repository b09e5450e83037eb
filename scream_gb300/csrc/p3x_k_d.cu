/* Column kernel instantiation: rate type double. */
#include "p3x_kernels_impl.cuh"

namespace p3x {
template cudaError_t launch_p3_part<double>(const dev::Inst&, const dev::KParams<double>&,
                                                 const LaunchSpec&, int, int, cudaStream_t);
}  // namespace p3x
