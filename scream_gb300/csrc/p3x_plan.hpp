/*
 * Sizes of the column kernels' launches: how many CTAs a launch may keep on the
 * GPU, when part1+2 takes a CTA per column, and the pools of columns that it
 * takes otherwise.  Plain integer code, for the host and the kernels.
 */
#ifndef P3X_PLAN_HPP
#define P3X_PLAN_HPP

#ifdef __CUDACC__
#define P3X_PLAN_HD __host__ __device__ __forceinline__
#else
#define P3X_PLAN_HD inline
#endif

namespace p3x {

namespace dev {
/* K1: level lists of a pool of columns, entries (column of the pool, level) */
constexpr int kPoolTiers = 5; /* pools of 16, 8, 4, 2, 1 columns */
constexpr int kPoolMaxCols = 1 << (kPoolTiers - 1);

/* Pool i of a launch's work items: pool_cols of them, and half as many whenever
 * the pools of a size are used up (pool_end), so that the last pools of a call of
 * several rounds are small and every warp ends at about the same time. */
template <class KP>
P3X_PLAN_HD void pool_range(const KP& kp, const int i, int& w0, int& w1) {
  int first = 0, size = kp.pool_cols;
  w0 = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int t = 0; t < kPoolTiers - 1; ++t) {
    if (i < kp.pool_end[t] || size == 1) break;
    w0 += (kp.pool_end[t] - first) * size;
    first = kp.pool_end[t];
    size >>= 1;
  }
  w0 += (i - first) * size;
  w1 = w0 + size < kp.nwork ? w0 + size : kp.nwork;
}
}  // namespace dev

/* CTAs that a persistent launch may keep resident: `per_sm` on each SM, at most
 * blocks_per_sm of them where that is given, and of all those the share
 * grid_frac (the rest stays free for other streams' launches). */
inline long long resident_ctas(int per_sm, int blocks_per_sm, int num_sms, double grid_frac) {
  if (blocks_per_sm > 0) per_sm = per_sm < blocks_per_sm ? per_sm : blocks_per_sm;
  long long grid = (long long)per_sm * num_sms;
  if (grid_frac > 0 && grid_frac < 1) {
    const long long share = (long long)(double(grid) * grid_frac);
    grid = share > 0 ? share : 1;
  }
  return grid;
}

/* K1 with a CTA per column (p3x_k_dwide.cu, p3x_k_fwide.cu): where all those
 * CTAs may be resident at once, at 2 an SM in the FP64 form, 4 in the FP32-bulk
 * form.  Measured, CTA per column against pools: 64 x 72 FP64 88 / 119 us, 304 x
 * 128 98 / 182, 456 x 128 183 / 182; FP32-bulk 64 x 72 22 / 32, 304 x 128 24 / 43. */
template <class TR>
inline bool part12_wide_fits(int nwork, int blocks_per_sm, int num_sms, double grid_frac) {
  return nwork <= resident_ctas(sizeof(TR) == sizeof(float) ? 4 : 2, blocks_per_sm, num_sms, grid_frac);
}

/* Columns of K1's largest pools: as many as have kPoolLevels levels (16 columns
 * of 128), 2 or 4 times as many at 16 or 8 lanes per column. */
constexpr int kPoolLevels = 2048;
inline int pool_columns(int nlev_max, int lanes) {
  int cols = 1;
  while (cols < dev::kPoolMaxCols && cols * 2 * nlev_max <= kPoolLevels) cols *= 2;
  for (int l = 32; l > lanes && cols < dev::kPoolMaxCols; l /= 2) cols *= 2;
  return cols;
}

/* Pools of K1 (pool_range) for `warps` resident warps.  A call of at most
 * pool_columns columns a warp gives every warp one pool of its share: against
 * pools that get smaller towards the end 2,600 x 72 FP64 271 us / 356, 5,400 x 72
 * 474 / 504, 16,000 x 128 1.86 ms / 1.99, FP32-bulk 16,000 x 128 262 us / 288.  A
 * larger call takes pools of C = pool_columns columns until C / 2 columns are left
 * for each warp, and then pools of half as many, and so on, and so does a work
 * list, whose instances differ in depth.  345,600 x 128 FP32-bulk: C = 16 4.86 ms,
 * 8 4.92, 4 5.33; the last pools from C / 4 or C columns a warp on instead of C /
 * 2: 86,400 x 128 FP32-bulk 1.34 and 1.32 ms against 1.30, after four steps
 * (nearly every level with a hydrometeor) 3.14 and 3.06 against 3.04; 43,200 x 128
 * FP64 4.58 and 4.74 against 4.53. */
template <class KP>
inline void plan_pools(KP& kp, int lanes, long long warps) {
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

}  // namespace p3x

#endif
