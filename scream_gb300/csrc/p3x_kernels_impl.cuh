/* Launch helpers of the column kernels (included by the per-variant TUs). */
#pragma once

#include "p3x_launch.hpp"

namespace p3x {

/* Persistent launch of one kernel: the grid is the number of CTAs that fit on
 * all SMs at once (capped by blocks_per_sm when given, and by what `groups`
 * groups of work need); groups walk the work list with a grid stride.  The occupancy comes
 * from a per-device cache, so a launch makes no attribute or occupancy query
 * after the first one of its shape. */
template <class TR, class Kern>
cudaError_t launch_persistent(Kern kern, const dev::Inst& inst0, const dev::KParams<TR>& kp, int threads,
                              size_t smem, int blocks_per_sm, int num_sms, cudaStream_t stream,
                              double grid_frac, long long groups) {
  int per_sm = 0;
  cudaError_t e = kernel_occupancy(reinterpret_cast<const void*>(kern), threads, smem, &per_sm);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidConfiguration;
  if (blocks_per_sm > 0) per_sm = per_sm < blocks_per_sm ? per_sm : blocks_per_sm;
  long long grid = (long long)per_sm * num_sms;
  /* a share of the capacity leaves room on every SM for other streams' launches */
  if (grid_frac > 0 && grid_frac < 1) {
    const long long share = (long long)(double(grid) * grid_frac);
    grid = share > 0 ? share : 1;
  }
  const long long need = (groups + kp.groups_per_block - 1) / kp.groups_per_block;
  if (need < grid) grid = need;
  if (grid <= 0) return cudaSuccess;
  kern<<<int(grid), threads, smem, stream>>>(inst0, kp);
  return cudaGetLastError();
}

/* Pools of K1 (pool_range).  A call of at most pool_columns columns for each of
 * the `warps` warps gives every warp one pool of its share: against pools that
 * get smaller towards the end 2,600 x 72 FP64 271 us / 356, 5,400 x 72 474 / 504,
 * 16,000 x 128 1.86 ms / 1.99, FP32-bulk 16,000 x 128 262 us / 288.  A larger call
 * takes pools of C = pool_columns columns until C / 2 columns are left for each
 * warp, and then pools of half as many, and so on, and so does a work list, whose
 * instances differ in depth.  345,600 x 128 FP32-bulk: C = 16 4.86 ms, 8 4.92, 4
 * 5.33; the last pools from C / 4 or C columns a warp on instead of C / 2: 86,400 x
 * 128 FP32-bulk 1.34 and 1.32 ms against 1.30, after four steps (nearly every level
 * with a hydrometeor) 3.14 and 3.06 against 3.04; 43,200 x 128 FP64 4.58 and 4.74
 * against 4.53. */
template <class TR>
void plan_pools(dev::KParams<TR>& kp, int lanes, long long warps) {
  int cols = pool_columns(kp.nlev_max, lanes);
  const long long share = (kp.nwork + warps - 1) / warps;
  const bool one_round = !kp.work && share <= cols;
  if (one_round) {
    cols = int(share);
  } else {
    while (cols > 2 && cols * warps > kp.nwork) cols /= 2;
    if (kp.nwork <= warps) cols = 1;
  }
  kp.pool_cols = cols;
  long long left = kp.nwork, n = 0;
  int t = 0;
  for (; cols > 1; cols /= 2) {
    const long long keep = one_round ? 0 : warps * cols / 2;
    const long long take = left > keep ? (left - keep + cols - 1) / cols : 0;
    n += take;
    left -= take * cols < left ? take * cols : left;
    kp.pool_end[t++] = int(n);
  }
  n += left;
  for (; t < dev::kPoolTiers - 1; ++t) kp.pool_end[t] = int(n);
  kp.npools = int(n);
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
    const bool wide = !ls.staged && part12_wide_fits<TR>(kp, num_sms); /* it zeroes the counters itself */
    if (kp.wctr && !wide) {
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
      const long long warps = (long long)per_sm * num_sms * kp.groups_per_block;
      plan_pools(kp, ls.lanes, warps);
      /* Fewer pools than warps: CTAs of one warp spread them evenly over the SMs
       * (912 x 97 FP64: CTAs of 4 warps 193 us, of 2 158). */
      int cta = threads;
      if (!ls.staged && kp.npools <= warps) {
        smem /= kp.groups_per_block;
        kp.groups_per_block = 1;
        cta = 32;
      }
      e = launch_persistent<TR>(kern, inst0, kp, cta, smem, ls.blocks_per_sm, num_sms, stream, ls.grid_frac, kp.npools);
    }
    if (e == cudaSuccess && ls.marks) cudaEventRecord(ls.marks[1], stream);
  } else if (part == kPartK2) {
    {
      const int wide = kp.wctr ? sed_wide_lanes(kp.nwork, kp.nlev_max, num_sms) : 0;
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
