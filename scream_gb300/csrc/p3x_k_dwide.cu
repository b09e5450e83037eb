/* Part1+2 and sedimentation with a CTA per column: rate type double.  Sedimentation
 * of at most one column an SM: the three species at once, in 128 threads each. */
#include "p3x_kernels_impl.cuh"

namespace p3x {
template <>
cudaError_t launch_part12_wide<double>(const dev::Inst& inst0, const dev::KParams<double>& kp,
                                        cudaStream_t stream) {
  const size_t smem = dev::pool_list_entries(1, kp.nlev_max) * sizeof(uint16_t) +
                      dev::kPreFields * sizeof(double) * size_t(kp.nlev_max < dev::kPreLevels ? kp.nlev_max : dev::kPreLevels);
  dev::p3_part12_wide_kernel<double><<<kp.nwork, dev::kPart12WideThreads, smem, stream>>>(inst0, kp);
  return cudaGetLastError();
}

template <>
cudaError_t launch_sed_wide<double>(const dev::Inst& inst0, const dev::KParams<double>& kp, int lanes, int num_sms,
                                cudaStream_t stream) {
  const size_t group =
      sizeof(dev::GroupScratch) + size_t(dev::sed_slots<double>()) * size_t(kp.sm_stride) * sizeof(double);
  if (lanes == 128 && kp.nwork <= num_sms) {
    dev::p3_sed_wide_kernel<128, true><<<kp.nwork, 384, 3 * group, stream>>>(inst0, kp);
  } else if (lanes == 128) {
    dev::p3_sed_wide_kernel<128, false><<<kp.nwork, 128, group, stream>>>(inst0, kp);
  } else {
    dev::p3_sed_wide_kernel<256, false><<<kp.nwork, 256, group, stream>>>(inst0, kp);
  }
  return cudaGetLastError();
}
}  // namespace p3x
