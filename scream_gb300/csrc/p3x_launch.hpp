/* Host-side launch interface of the device kernels (internal to libp3x). */
#ifndef P3X_LAUNCH_HPP
#define P3X_LAUNCH_HPP

#include <cuda_runtime.h>

#include "p3x.h"
#include "p3x_column.cuh"

struct p3x_context;

namespace p3x {

struct LaunchSpec {
  int lanes;            /* 8, 16, 32 */
  int groups_per_block; /* columns per CTA */
  int staged;           /* tables in shared memory */
  int blocks_per_sm;    /* part1+2: CTAs an SM at most; 0: as many as fit */
  cudaEvent_t* marks = nullptr; /* optional: 4 events recorded around K1, K2, K3 */
  double grid_frac = 1.0;       /* share of the resident-CTA capacity the persistent grid takes */
};

/* Threads of a CTA: the configured columns x lanes in whole warps. */
inline int warp_threads(const LaunchSpec& ls) { return (ls.groups_per_block * ls.lanes + 31) / 32 * 32; }

/* Shared-memory bytes of one CTA of K1 (part1+part2; staged tables plus the
 * level lists) and of K2 (sedimentation).  K3 uses none. */
template <class TR>
inline size_t p3_smem_bytes(const LaunchSpec& ls, int nlev_max) {
  const size_t tables = ls.staged ? dev::table_smem_bytes<TR>() : 0;
  return tables + size_t(warp_threads(ls) / 32) * dev::pool_list_entries(pool_columns(nlev_max, ls.lanes), nlev_max) *
                      sizeof(uint16_t);
}
template <class TR>
inline size_t sed_smem_bytes(const LaunchSpec& ls, int sm_stride) {
  return size_t(ls.groups_per_block) * dev::sed_slots<TR>() * size_t(sm_stride) * sizeof(double);
}

/* Launch shape of K2 and K3: always 32 lanes per column.  Sedimentation's
 * substeps walk the levels chunk by chunk, so a narrower group only lengthens the
 * walk (65,536 x 128 with 16 lanes: FP64 K2 +17 %, FP32-bulk K2 +95 %); part3 FP64
 * at 21,600 x 128 took 344 us with 32 lanes, 369 with 16.  Columns per CTA as
 * configured, at most 8 (256 threads). */
inline LaunchSpec sed_spec(const LaunchSpec& ls) {
  LaunchSpec s = ls;
  s.lanes = 32;
  s.groups_per_block = ls.groups_per_block < 8 ? ls.groups_per_block : 8;
  s.staged = 0;
  return s;
}

/* Threads per column of K2 where a call leaves most warps idle: a CTA of 128
 * or 256 threads (at least the column's levels) per column while at most 32
 * warps an SM result; 0: 32 lanes per column.  Measured, CTA per column against
 * 32 lanes: 608 x 128 FP64 220 / 351 us, FP32-bulk 82 / 140; 1,216 x 128 330 /
 * 388 and 109 / 156; 1,520 x 72 213 / 180 and 85 / 75. */
inline int sed_wide_lanes(int nwork, int nlev_max, int num_sms) {
  const int lanes = nlev_max <= 128 ? 128 : (nlev_max <= 256 ? 256 : 0);
  return lanes && nlev_max > 32 && (long long)nwork * (lanes / 32) <= (long long)num_sms * 32 ? lanes : 0;
}
/* Launch of K2 with a CTA per column (p3x_k_dwide.cu, p3x_k_fwide.cu). */
template <class TR>
cudaError_t launch_sed_wide(const dev::Inst& inst0, const dev::KParams<TR>& kp, int lanes, int num_sms,
                            cudaStream_t stream);

/* K1 with a CTA per column (part12_wide_fits). */
template <class TR>
cudaError_t launch_part12_wide(const dev::Inst& inst0, const dev::KParams<TR>& kp, cudaStream_t stream);

/* Columns of one CTA of the FP32-bulk sedimentation that keeps its tables in
 * shared memory, one CTA per SM: as many as fit beside the 20.8 KB of tables, 20
 * at most (96 registers a thread).  0 where that is fewer than 16. */
inline int sed_staged_columns(int sm_stride) {
  const size_t col = dev::kSedBulkSlots * size_t(sm_stride) * sizeof(double);
  const size_t n = (size_t(227 * 1024) - dev::sed_table_bytes()) / col;
  return n >= 20 ? 20 : (n >= 16 ? int(n) : 0);
}

/* CTAs of kernel `func` that fit on one SM with `threads` threads and `smem`
 * bytes of dynamic shared memory on the current device.  The first query of
 * a (device, kernel, threads, smem) shape raises the kernel's
 * dynamic-shared-memory limit as needed and asks the occupancy calculator;
 * later ones read the cache (p3x_api.cu). */
cudaError_t kernel_occupancy(const void* func, int threads, size_t smem, int* per_sm);

/* Kernel parts of one step, launched in order on one stream: K1
 * (part1+part2; zeroes the work counters first), K2 (sedimentation), K3
 * (part3). */
enum : int { kPartK1 = 1, kPartK2 = 2, kPartK3 = 4 };

/* Persistent launch of one part (defined in p3x_kernels_impl.cuh, instantiated
 * in p3x_k_d.cu and p3x_k_f.cu).
 * kp.nwork, kp.work, kp.insts and kp.sm_stride are set by the caller, and
 * every instance's scratch (Inst::scr, Inst::cflag) is bound. */
template <class TR>
cudaError_t launch_p3_part(const dev::Inst& inst0, const dev::KParams<TR>& kp, const LaunchSpec& ls, int part,
                           int num_sms, cudaStream_t stream);

/* The column kernels of one step in order on one stream: all three (K1, K2,
 * K3) by default, or the subset `parts` (kPartK* bits).  K1 zeroes the work
 * counters; a subset without K1 zeroes them here. */
template <class TR>
inline cudaError_t launch_p3(const dev::Inst& inst0, const dev::KParams<TR>& kp, const LaunchSpec& ls,
                             int num_sms, cudaStream_t stream, int parts = kPartK1 | kPartK2 | kPartK3) {
  cudaError_t e = cudaSuccess;
  if (parts & kPartK1) {
    e = launch_p3_part<TR>(inst0, kp, ls, kPartK1, num_sms, stream);
    if (e != cudaSuccess) return e;
  } else if (kp.wctr) {
    e = cudaMemsetAsync(kp.wctr, 0, dev::kWorkCounters * sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
  }
  if (parts & kPartK2) {
    e = launch_p3_part<TR>(inst0, kp, sed_spec(ls), kPartK2, num_sms, stream);
    if (e != cudaSuccess) return e;
  }
  if (parts & kPartK3) e = launch_p3_part<TR>(inst0, kp, sed_spec(ls), kPartK3, num_sms, stream);
  return e;
}

/* (nlev, ncol) column-fastest <-> (ncol, ld) level-contiguous transposes. */
cudaError_t launch_transpose_to_levels(const double* src, double* dst, int ncol, int nlev, int64_t ld,
                                       cudaStream_t st);
cudaError_t launch_transpose_to_columns(const double* src, double* dst, int ncol, int nlev, int64_t ld,
                                        cudaStream_t st);

/* One step of a work list of (instance, column) items, each column once and in
 * any order (dev::WorkItem), whose instances all have the given precision: K1,
 * K2, K3 with the context's launch configuration for that precision
 * (p3x_api.cu).  Every instance's scratch must be bound.  wctr:
 * dev::kWorkCounters device words used by no other launch in flight (zeroed on
 * the stream), or null for a static stride. */
int launch_work(p3x_context* ctx, const p3x_runtime& rt, int precision, const dev::Inst* insts_d,
                const dev::WorkItem* work_d, int nwork, int nlev_max, uint32_t* wctr, cudaStream_t st,
                double grid_frac = 1.0);

/* The state hand-over of the P3 process interface between steps
 * (eamxx_p3_process_interface.hpp:218,237 with dry = wet mixing ratios):
 * qv_prev <- qv and t_prev <- th / inv_exner, for every work item. */
cudaError_t launch_postamble(const dev::Inst* insts_d, const dev::WorkItem* work_d, int nwork, cudaStream_t st);

/* Device pointers of the process-interface pre/postamble kernels. */
struct InterfacePtrs {
  const double *pmid, *pd, *pdd, *cld_t;
  double *T, *T_prev;
  double* q[9]; /* qc nc qr nr qi qm ni bm qv */
  double *th, *qv_prev, *inv_exner, *dz, *cld_l, *cld_i, *cld_r;
  double *eff_qc, *eff_qi, *eff_qr;
  const double *liq_surf, *ice_surf;
  double *liq_mass, *ice_mass, *vapor_flux, *water_flux, *ice_flux, *heat_flux;
};
cudaError_t launch_interface(const InterfacePtrs& p, int ncol, int nlev, int64_t ld, bool post, double dt,
                             cudaStream_t st);

/* Device pointers of the EAM driver's pre/post kernels (micro_p3_tend).
 * Constituent order of q, ptend_q and w: qv, cldliq, numliq, rain, numrain,
 * cldice, numice, cldrim, rimvol. */
struct EamPtrs {
  const double *pmid, *pmiddry, *pdel, *pdeldry, *zi, *t, *q[9], *ast, *npccn, *ni_act_in, *relvar, *cmeliq;
  double *t_prev, *qv_prev, *ptend_s, *ptend_q[9];
  double *qme, *rho, *icimrst, *icwmrst, *icinc, *icwnc, *rel, *rei, *dei, *mu, *lambdac, *nfice, *efcout, *ncout,
      *freql, *efiout, *niout, *freqi, *aqrain, *anrain, *freqr, *reff_rain, *deff_rain, *flxprc, *flxsnw;
  double *prec_pcw, *snow_pcw, *prec_str, *snow_str, *cdnumc;
  int subgrid, method;
  /* the P3 working arrays: prognostic state in constituent order, inputs */
  double* w[9];
  double *th, *pres, *dz, *dpres, *inv_exner, *cld_l, *cld_i, *cld_r, *nc_nuceat, *ni_act, *inv_relvar, *qv_prev_dry,
      *t_prev_p3;
  /* P3 outputs read by the post kernel */
  const double *eff_qc, *eff_qi, *eff_qr, *liq_surf, *ice_surf, *liq_flux, *ice_flux, *depos;
  double* vap_liq;
};
cudaError_t launch_eam(const EamPtrs& p, int ncol, int nlev, int64_t ld, int64_t ld_int, bool post, double dt,
                       cudaStream_t st);

/* Murphy-Koop vapour pressure over liquid at 0 C, evaluated on the device
 * (synchronous). */
cudaError_t saturation_at_melting(double* out);

cudaError_t launch_selftest(unsigned long long* mismatches_d, cudaStream_t st);
/* The device's words of the fixed-point self-test (p3x_fixtest.hpp). */
cudaError_t launch_fix_selftest(const int64_t* coef_d, uint64_t* out_d, cudaStream_t st);

/* Fields of the column mass / energy conservation check (device pointers;
 * per-level (ncol, ld), winds (ncol, 2, ld), per-column (ncol)). */
struct ConsPtrs {
  const double *pd, *T, *qv, *qc, *qi, *qr, *winds, *ps, *phis;
  const double *vapor_flux, *water_flux, *ice_flux, *heat_flux;
  double *mass, *energy;                    /* column totals (may be null)   */
  const double *mass_before, *energy_before; /* null: totals only            */
  double *mass_err, *energy_err;            /* relative errors (with before) */
};
/* Column totals and, with the totals before, relative errors; with maxloc4
 * (4 doubles, device), also {max mass err, its column, max energy err, its
 * column}. */
cudaError_t launch_conservation(const ConsPtrs& p, int ncol, int nlev, int64_t ld, double dt, double* maxloc4,
                                cudaStream_t st);

cudaError_t launch_budgets(const double* qv, const double* qc, const double* qr, const double* qi,
                           const double* th, const double* dpres, const double* inv_exner, int ncol,
                           int nlev, int64_t ld, double* water, double* energy, cudaStream_t st);

}  // namespace p3x

#endif
