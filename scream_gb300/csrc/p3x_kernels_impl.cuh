/* Launch helpers of the column kernels (included by the per-variant TUs). */
#pragma once

#include "p3x_launch.hpp"

namespace p3x {

/* Persistent launch of one kernel: the grid is the number of CTAs that may be
 * resident at once (resident_ctas), or what `groups` groups of work need; groups
 * walk the work list with a grid stride.  The occupancy comes from a per-device
 * cache, so a launch makes no attribute or occupancy query after the first one of
 * its shape. */
template <class TR, class Kern>
cudaError_t launch_persistent(Kern kern, const dev::Inst& inst0, const dev::KParams<TR>& kp, int threads,
                              size_t smem, int blocks_per_sm, int num_sms, cudaStream_t stream,
                              double grid_frac, long long groups) {
  int per_sm = 0;
  cudaError_t e = kernel_occupancy(reinterpret_cast<const void*>(kern), threads, smem, &per_sm);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidConfiguration;
  long long grid = resident_ctas(per_sm, blocks_per_sm, num_sms, grid_frac);
  const long long need = (groups + kp.groups_per_block - 1) / kp.groups_per_block;
  if (need < grid) grid = need;
  if (grid <= 0) return cudaSuccess;
  kern<<<int(grid), threads, smem, stream>>>(inst0, kp);
  return cudaGetLastError();
}

template <class TR>
cudaError_t launch_p3_part(const dev::Inst& inst0, const dev::KParams<TR>& kp_in, const LaunchSpec& ls, int part,
                           int num_sms, cudaStream_t stream) {
  constexpr int LANES = 32;
  dev::KParams<TR> kp = kp_in;
  const int threads = warp_threads(ls);
  kp.groups_per_block = threads / 32;
  kp.staged = ls.staged;
  cudaError_t e = cudaErrorInvalidValue;
  if (part == kPartK1) {
    const bool wide = !ls.staged && part12_wide_fits<TR>(kp.nwork, ls.blocks_per_sm, num_sms, ls.grid_frac);
    if (kp.wctr && !wide) { /* the kernel with a CTA per column zeroes them itself */
      e = cudaMemsetAsync(kp.wctr, 0, dev::kWorkCounters * sizeof(uint32_t), stream);
      if (e != cudaSuccess) return e;
    }
    if (ls.marks) cudaEventRecord(ls.marks[0], stream);
    if (wide) {
      e = launch_part12_wide<TR>(inst0, kp, stream);
    } else {
      const auto kern = kp.work ? dev::p3_part12_kernel<TR, true> : dev::p3_part12_kernel<TR, false>;
      size_t smem = p3_smem_bytes<TR>(ls, kp.nlev_max);
      int per_sm = 0;
      e = kernel_occupancy(reinterpret_cast<const void*>(kern), threads, smem, &per_sm);
      if (e != cudaSuccess) return e;
      if (per_sm <= 0) return cudaErrorInvalidConfiguration;
      const long long warps =
          resident_ctas(per_sm, ls.blocks_per_sm, num_sms, ls.grid_frac) * kp.groups_per_block;
      plan_pools(kp, ls.lanes, warps);
      /* Fewer pools than warps: CTAs of one warp spread them evenly over the SMs
       * (912 x 97 FP64: CTAs of 4 warps 193 us, of 2 158), where as many of those
       * may be resident. */
      int cta = threads;
      if (!ls.staged && kp.npools <= warps) {
        const size_t warp_smem = smem / kp.groups_per_block;
        e = kernel_occupancy(reinterpret_cast<const void*>(kern), 32, warp_smem, &per_sm);
        if (e != cudaSuccess) return e;
        if (kp.npools <= resident_ctas(per_sm, ls.blocks_per_sm, num_sms, ls.grid_frac)) {
          smem = warp_smem;
          kp.groups_per_block = 1;
          cta = 32;
        }
      }
      e = launch_persistent<TR>(kern, inst0, kp, cta, smem, ls.blocks_per_sm, num_sms, stream, ls.grid_frac, kp.npools);
    }
    if (e == cudaSuccess && ls.marks) cudaEventRecord(ls.marks[1], stream);
  } else if (part == kPartK2) {
    {
      const int wide = kp.wctr && ls.grid_frac >= 1 ? sed_wide_lanes(kp.nwork, kp.nlev_max, num_sms) : 0;
      if (wide) {
        e = launch_sed_wide<TR>(inst0, kp, wide, num_sms, stream);
      } else if constexpr (sizeof(TR) == sizeof(float)) {
        const int per_sm = sed_staged_columns(kp.sm_stride);
        if (kp.wctr && per_sm > 0 && kp.nwork >= per_sm * num_sms) {
          kp.groups_per_block = per_sm;
          const size_t smem = dev::sed_table_bytes() +
                              size_t(per_sm) * dev::kSedBulkSlots * size_t(kp.sm_stride) * sizeof(double);
          e = launch_persistent<TR>(dev::p3_sed_bulk_kernel<LANES, true>, inst0, kp, per_sm * LANES, smem, 0, num_sms,
                                    stream, ls.grid_frac, kp.nwork);
        } else {
          e = launch_persistent<TR>(dev::p3_sed_bulk_kernel<LANES, false>, inst0, kp, threads,
                                    sed_smem_bytes<TR>(ls, kp.sm_stride), 0, num_sms, stream, ls.grid_frac, kp.nwork);
        }
      } else {
        e = launch_persistent<TR>(dev::p3_sed_kernel<TR, LANES>, inst0, kp, threads,
                                  sed_smem_bytes<TR>(ls, kp.sm_stride), 0, num_sms, stream, ls.grid_frac, kp.nwork);
      }
      if (e == cudaSuccess && ls.marks) cudaEventRecord(ls.marks[2], stream);
    }
  } else if (part == kPartK3) {
    {
      /* Levels are independent here: where the columns leave warps idle, one
       * warp takes 32 levels of a column instead of all of them (64 x 72: FP64
       * 31 -> 16 us, FP32-bulk 16 -> 10 us). */
      const auto kern = dev::p3_part3_kernel<TR, LANES>;
      int per_sm = 0;
      e = kernel_occupancy(reinterpret_cast<const void*>(kern), threads, 0, &per_sm);
      if (e != cudaSuccess) return e;
      const int chunks = (kp.sm_stride - 1 + LANES - 1) / LANES;
      const long long groups = (long long)per_sm * num_sms * kp.groups_per_block;
      kp.part3_split = kp.wctr && (long long)kp.nwork * chunks <= groups ? chunks : 1;
      e = launch_persistent<TR>(kern, inst0, kp, threads, 0, 0, num_sms, stream, ls.grid_frac,
                                (long long)kp.nwork * kp.part3_split);
      if (e == cudaSuccess && ls.marks) cudaEventRecord(ls.marks[3], stream);
    }
  }
  return e;
}

}  // namespace p3x
