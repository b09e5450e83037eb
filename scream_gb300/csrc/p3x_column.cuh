/*
 * The P3 step as three column kernels.
 *
 * Inputs are level-contiguous (EAMxx layout): the lanes of a warp take
 * neighbouring levels, so loads of one field are coalesced.  The reference's
 * stage order (p3/impl/p3_main_impl.hpp:108-325) is kept across three launches
 * on one stream:
 *
 *   K1 p3_part12_kernel: p3_main_init + p3_main_part1 and p3_main_part2
 *      (level-parallel; a warp takes a pool of columns, a CTA one column where
 *      a call is small), with the two column-wide early exits of
 *      p3_main_impl.hpp:237-239 and :260.  It hands the per-level
 *      start-of-step temperature, density and fall-speed factors to K2/K3
 *      through a scratch array and marks each column that goes on.
 *   K2 p3_sed_kernel: cloud, rain and ice sedimentation, a column to a warp or,
 *      where a call is small, to a CTA: CFL substeps with the Courant maximum
 *      as a group reduction and the upwind flux divergence walked down the
 *      levels chunk by chunk with a shuffle-up and a carry
 *      (p3_upwind_impl.hpp:14-116).  Substep loops are capped.
 *   K3 p3_part3_kernel: homogeneous freezing + p3_main_part3.
 *
 * Splitting lets each kernel keep its own register and shared-memory
 * footprint: part2's ~45 rates no longer limit the occupancy of the
 * latency-bound sedimentation walk.  K1 keeps only its level lists in shared
 * memory, K2 its per-level arrays (9 or 10 slots of FP64 width per column).
 * Lookup tables are read from global memory (L1/L2) or, in K1, staged into
 * shared memory once per CTA with cp.async.bulk + mbarrier (Table3 slices for
 * the runtime's constant rain shape parameter, plus the whole ice table).
 */
#pragma once

#include <type_traits>

#include "p3x_physics.cuh"
#include "p3x_plan.hpp"

namespace p3x {
namespace dev {

/* Arguments of one instance (device pointers, (ncol, nlev) row-major). */
struct Inst {
  double *qc, *nc, *qr, *nr, *qi, *qm, *ni, *bm, *qv, *th;
  const double *nc_nuceat_tend, *nccn, *ni_activated, *inv_qc_relvar, *cld_frac_i, *cld_frac_l,
      *cld_frac_r, *pres, *dz, *dpres, *inv_exner, *qv_prev, *t_prev;
  double *qv2qi_depos_tend, *precip_liq_surf, *precip_ice_surf, *diag_eff_radius_qc,
      *diag_eff_radius_qi, *diag_eff_radius_qr, *rho_qi, *precip_liq_flux, *precip_ice_flux,
      *precip_total_tend, *nevapr;
  double *liq_ice_exchange, *vap_liq_exchange, *vap_ice_exchange;
  /* hand-over from K1 to K2/K3: [kScrFields][ncol][ld] doubles, and one
   * continue flag per column (0: the column took an early exit) */
  double* scr;
  int32_t* cflag;
  int64_t ld, ld_int;
  int32_t ncol, nlev;
  double dt;
  int32_t predictNc, prescribedCCN, precision, pad_;
};

/* Work item of the batched form: (instance, column).  Any order gives the same
 * results; part1+2 pools neighbouring items that are neighbouring columns of one
 * instance (work_run), so lists hold an instance's columns in a row. */
struct WorkItem {
  int32_t inst, col;
};

constexpr int kPoolLevelBits = 12;
constexpr int kPart12WideThreads = 128;
/* what the warps of a CTA share where they work on one column */
struct PoolScratch {
  uint32_t n_hyd, n_nuc, active;
};
/* deeper columns than that do not fit K2's shared memory either */
static_assert(kPoolMaxCols << kPoolLevelBits == 1 << 16, "16-bit entries");
__host__ __device__ constexpr size_t pool_list_entries(int cols, int nlev_max) {
  return (size_t(cols) * size_t(nlev_max) + 7) / 8 * 8;
}

template <class TR>
struct KParams {
  RuntimeDev rt;
  /* global tables in the rate precision */
  const TR* ice;
  const TR* ice_sed; /* FP32-bulk: slots 0-3 of every ice-table row, packed */
  const TR* collect;
  const TR* vn;
  const TR* vm;
  const TR* revap;
  /* FP64 form: the fixed-point ice-table cells of sedimentation (columns 0, 1, 6, 7) and
   * part3 (6, 7, 5, 11) with their powers of two, and Table3's fall speeds as
   * {vm, vm step, vn, vn step} per row for each of the 10 mu columns */
  const int64_t *cell_sed, *cell_part3;
  const int32_t *cell_sed_shift, *cell_part3_shift;
  const double4* t3sed;
  const TR* t3slice; /* [3][300][2] = vn, vm, revap columns (t3_dumjj-1, t3_dumjj) */
  int staged;        /* stage ice table + Table3 slices into shared memory */
  int sm_stride;     /* doubles per per-level shared array (>= nlev_max + 1, even) */
  int groups_per_block;
  int nwork;         /* number of columns (single) or work items (batched) */
  int nlev_max;      /* levels of the deepest column */
  int part3_split;   /* K3: groups that share a work item's levels */
  int pool_cols;     /* K1: columns of the largest pool */
  int npools;        /* K1: pools */
  int pool_end[kPoolTiers - 1]; /* K1: pools of pool_cols columns, of those and half that, ... (running totals) */
  const WorkItem* work;
  const Inst* insts;
  uint32_t* err;
  double esat0; /* liquid saturation vapour pressure at 0 C (ice_melting, ice_cldliq_wet_growth) */
  /* kWorkCounters zeroed counters: groups take work items from them as they
   * finish the last ones.  Null: groups stride the list statically. */
  uint32_t* wctr;
  /* check_values after part3 (null: off): kCheckWords words of CheckWord */
  unsigned long long* check;
  int check_fail; /* a temperature out of range also sets kErrRange */
};

/* check_values (p3_check_values_impl.hpp): counts of levels with T outside
 * (173, 323) K and with qv outside (0, 0.04), and the smallest packed
 * (instance, column, level) key of each kind. */
enum CheckWord { kChkTCount = 0, kChkQvCount, kChkTFirst, kChkQvFirst, kCheckWords };
__host__ __device__ inline unsigned long long check_key(int inst, int col, int k) {
  return (static_cast<unsigned long long>(inst) << 40) | (static_cast<unsigned long long>(col) << 16) |
         static_cast<unsigned long long>(k);
}

constexpr int kIceTableElems = kDensize * kRimsize * kIsize * kIceCols; /* 12000 */
constexpr int kT3SliceElems = 3 * 300 * 2;
constexpr int kSedIceElems = kDensize * kRimsize * kIsize * kIceSedCols; /* 4000 */
/* shared bytes of the FP32-bulk sedimentation's staged tables */
__host__ __device__ constexpr size_t sed_table_bytes() {
  return sizeof(float) * (kSedIceElems + 2 * (kT3SliceElems / 3));
}
constexpr int kT3SedRows = 300;
/* (RHO_600MB / RHO_1000MB)^0.54 */
constexpr double kRhofaciOverR = 0.790740972875368752906;
constexpr long long kInfBits = 0x7ff0000000000000ll;
constexpr uint64_t kNaNBits = 0x7ff8000000000000ull;
constexpr int kMaxSubsteps = 100000;
constexpr long long kWaitSpinLimit = 1ll << 26;
constexpr uint64_t kWaitNanosLimit = 2000000000ull; /* 2 s */

/* shared arrays of one column group in K2 (FP64 form, p3_sed); the rain flux
 * accumulator re-uses R2 (rain has two fields) */
enum { B_FR = 0, B_CF, B_QS, B_V1, B_V2, B_R0, B_R1, B_R2, B_R3, B_NARR };
/* slots (of S doubles) of one column group in K2: B_NARR in the FP64 form,
 * kSedBulkSlots in the FP32-bulk form (p3_sed_bulk) */
constexpr int kSedBulkSlots = 10;
template <class TR>
__host__ __device__ constexpr int sed_slots() {
  return sizeof(TR) == sizeof(float) ? kSedBulkSlots : B_NARR;
}
/* hand-over fields K1 -> K2/K3 */
enum { S_TATM = 0, S_RHO, S_RHOFACR, S_RHOFACI, S_ACN, kScrFields };

__device__ __forceinline__ double* scr_at(const Inst& in, int f, int col) {
  return in.scr + (int64_t(f) * in.ncol + col) * in.ld;
}
/* FP32-bulk: the float-valued hand-over fields (rho, fall-speed factors,
 * acn) hold floats in the first half of each column's row */
__device__ __forceinline__ float* scr_f(const Inst& in, int f, int col) {
  return reinterpret_cast<float*>(scr_at(in, f, col));
}

/* a read where it stands */
template <class T>
__device__ __forceinline__ T read_now(const T* p) {
  return *const_cast<const volatile T*>(p);
}

/* Launch-wide work counters of one step (K1, K2, K3, spare), zeroed on the
 * stream before K1, or by a K1 that does not use them.  They follow the
 * hand-over doubles and the flags in an instance's scratch. */
constexpr int kWorkCounters = 4;
__host__ __device__ inline size_t work_counter_offset(int ncol, int64_t ld) {
  const size_t d = size_t(kScrFields) * size_t(ncol) * size_t(ld) * sizeof(double);
  return ((d + size_t(ncol) * sizeof(int32_t) + 15) / 16) * 16;
}
/* bytes of the K1->K2/K3 scratch of an instance (doubles, flags, counters) */
__host__ __device__ inline size_t scratch_bytes(int ncol, int64_t ld) {
  return ((work_counter_offset(ncol, ld) + kWorkCounters * sizeof(uint32_t) + 255) / 256) * 256;
}

template <class TR>
__host__ __device__ constexpr size_t table_smem_bytes() {
  return ((sizeof(TR) * (kIceTableElems + kT3SliceElems) + 15) / 16) * 16 + 16;
}

/* ------------------------------------------------------------------ */
/* group primitives                                                    */
/* ------------------------------------------------------------------ */
/* Maxima and minima over the group with the warp-reduction instruction
 * (redux.sync), one instruction instead of five dependent shuffles.
 * Non-negative floats and doubles order as their bit patterns (as unsigned
 * integers), so their maximum is the maximum of the patterns; a NaN (a
 * pattern above +inf) wins and reaches the caller's Courant check. */
/* maximum over the group of non-negative doubles (dmax_nn): the largest high
 * word, then the largest low word among the lanes holding it */
__device__ __forceinline__ double group_max_nn(unsigned mask, double v) {
  const unsigned hi = unsigned(__double2hiint(v)), lo = unsigned(__double2loint(v));
  const unsigned mhi = __reduce_max_sync(mask, hi);
  const unsigned mlo = __reduce_max_sync(mask, hi == mhi ? lo : 0u);
  return __hiloint2double(int(mhi), int(mlo));
}
/* maximum over the group of non-negative floats (Courant numbers) */
__device__ __forceinline__ float group_max_nn(unsigned mask, float v) {
  return __uint_as_float(__reduce_max_sync(mask, __float_as_uint(v)));
}
__device__ __forceinline__ int group_min_int(unsigned mask, int v) {
  return __reduce_min_sync(mask, v);
}
__device__ __forceinline__ int group_max_int(unsigned mask, int v) {
  return __reduce_max_sync(mask, v);
}

/* The lanes of a warp that hold the levels base to last, base + lane each (base
 * <= last): the mask of a vote in a loop over those levels. */
__device__ __forceinline__ unsigned chunk_mask(int base, int last) {
  const int n = last - base + 1;
  return n < 32 ? (1u << n) - 1u : 0xffffffffu;
}

/* A sedimentation group is a warp or several, LANES > 32 threads (at least
 * as many as the column has levels): the warps of a group exchange through this
 * shared scratch and meet at a barrier.  SPLIT: a CTA has three such groups,
 * one per species, each with its own scratch and barrier (named 1 to 3);
 * otherwise the group is the CTA. */
struct GroupScratch {
  double max_d[8];
  float max_f[8];
  int lo[3][8], hi[3][8]; /* tops and bottoms of the species */
  double edge[8][4];      /* fluxes of each warp's last level */
  double prt[4];          /* surface precipitation of the species */
};
static_assert(sizeof(GroupScratch) % 16 == 0, "the arrays behind it are 16-byte aligned");
template <int LANES, bool SPLIT = false>
__device__ __forceinline__ void group_sync(unsigned mask) {
  if constexpr (SPLIT) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + int(threadIdx.x) / LANES), "n"(LANES) : "memory");
  } else if constexpr (LANES > 32) {
    __syncthreads();
  } else {
    __syncwarp(mask);
  }
}
template <int LANES>
__device__ __forceinline__ int group_warp() {
  return int(threadIdx.x & (LANES - 1)) >> 5;
}
/* Tops (minima) and bottoms (maxima) of the three species over the group. */
template <int LANES, bool SPLIT>
__device__ __forceinline__ void group_bounds(unsigned mask, GroupScratch* gs, int lo[3], int hi[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    lo[i] = group_min_int(mask, lo[i]);
    hi[i] = group_max_int(mask, hi[i]);
  }
  if constexpr (LANES > 32) {
    const int w = group_warp<LANES>();
    if ((threadIdx.x & 31) == 0) {
      for (int i = 0; i < 3; ++i) {
        gs->lo[i][w] = lo[i];
        gs->hi[i][w] = hi[i];
      }
    }
    group_sync<LANES, SPLIT>(mask);
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < LANES / 32; ++j) {
        lo[i] = min(lo[i], gs->lo[i][j]);
        hi[i] = max(hi[i], gs->hi[i][j]);
      }
  }
}
/* maximum of non-negative values over the group */
template <int LANES, bool SPLIT>
__device__ __forceinline__ double group_max_wide(unsigned mask, GroupScratch* gs, double v) {
  v = group_max_nn(mask, v);
  if constexpr (LANES > 32) {
    if ((threadIdx.x & 31) == 0) gs->max_d[group_warp<LANES>()] = v;
    group_sync<LANES, SPLIT>(mask);
    for (int j = 0; j < LANES / 32; ++j) v = dmax_nn(v, gs->max_d[j]);
  }
  return v;
}
template <int LANES, bool SPLIT>
__device__ __forceinline__ float group_max_wide(unsigned mask, GroupScratch* gs, float v) {
  v = group_max_nn(mask, v);
  if constexpr (LANES > 32) {
    if ((threadIdx.x & 31) == 0) gs->max_f[group_warp<LANES>()] = v;
    group_sync<LANES, SPLIT>(mask);
    for (int j = 0; j < LANES / 32; ++j)
      v = __float_as_uint(v) < __float_as_uint(gs->max_f[j]) ? gs->max_f[j] : v;
  }
  return v;
}

/* ------------------------------------------------------------------ */
/* bulk copy of the tables into shared memory                          */
/* ------------------------------------------------------------------ */
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

/* Thread 0 arms an mbarrier with the byte count and issues the bulk copies;
 * every thread then waits on the barrier's phase with a bounded spin.
 * Returns false (and sets kErrWait) if the wait gave up. */
template <class TR>
__device__ bool stage_tables(const KParams<TR>& kp, TR* s_ice, TR* s_t3, uint64_t* mbar, uint32_t& err) {
  const uint32_t bar = smem_u32(mbar);
  const uint32_t ice_bytes = uint32_t(sizeof(TR) * kIceTableElems);
  const uint32_t t3_bytes = uint32_t(sizeof(TR) * kT3SliceElems);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"(ice_bytes + t3_bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(s_ice)),
        "l"(kp.ice), "r"(ice_bytes), "r"(bar)
        : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(s_t3)),
        "l"(kp.t3slice), "r"(t3_bytes), "r"(bar)
        : "memory");
  }
  bool done = false;
  uint64_t t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (long long spin = 0; spin < kWaitSpinLimit; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(0)
        : "memory");
    if (ok) {
      done = true;
      break;
    }
    uint64_t t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (t1 - t0 > kWaitNanosLimit) break;
  }
  if (!done) err |= kErrWait;
  return done;
}

/* Applies a rate-precision DSD adjustment of a number concentration to the
 * FP64 value only when the DSD routine changed it (exact for FP64). */
template <class TR>
__device__ __forceinline__ void apply_n_adjust(double& n_d, TR n_in, TR n_out) {
  if (n_out != n_in) n_d = double(n_out);
}

/* The end of p3_main_part2 (p3_main_part2_impl.hpp, after update_prognostics):
 * a species below qsmall goes to vapour and its latent heat to theta; a +0
 * moves nothing, so its FP64 updates are skipped (bitwise the same result).
 * Returns whether any species remains. */
__device__ __forceinline__ bool clip_to_vapour(State& s, double inv_exner) {
  bool hydro = false;
  if (dlt(s.qc, C::QSMALL)) {
    if (dnz(s.qc)) {
      s.qv = s.qv + s.qc;
      s.th = s.th - inv_exner * s.qc * C::LatVap * C::INV_CP;
    }
    s.qc = 0;
    s.nc = 0;
  } else {
    hydro = true;
  }
  if (dlt(s.qr, C::QSMALL)) {
    if (dnz(s.qr)) {
      s.qv = s.qv + s.qr;
      s.th = s.th - inv_exner * s.qr * C::LatVap * C::INV_CP;
    }
    s.qr = 0;
    s.nr = 0;
  } else {
    hydro = true;
  }
  if (dlt(s.qi, C::QSMALL)) {
    if (dnz(s.qi)) {
      s.qv = s.qv + s.qi;
      s.th = s.th - inv_exner * s.qi * (C::LatVap + C::LatIce) * C::INV_CP;
    }
    s.qi = 0; s.ni = 0; s.qm = 0; s.bm = 0;
  } else {
    hydro = true;
  }
  return hydro;
}

/* Whether a level without hydrometeors below freezing may nucleate ice, which
 * takes T < Tmelt - 15 and a supersaturation over ice of 0.05.  The FP32
 * Murphy-Koop formula is good to 1e-4 of the ratio and the margin is ten times
 * that; true wherever FP32 cannot exclude it (also below 150 K and for NaN). */
__device__ __forceinline__ bool may_nucleate(double T, float tf, float qv, float p) {
  if (dgt(T, C::Tmelt - 14.9)) return false;
  const float e = __expf(9.550426f - 5723.265f / tf + 3.53068f * __logf(tf) - 0.00728332f * tf);
  return !(dgt(T, 150.0) && qv * p / (float(C::ep_2) * e) - 1.0f < 0.049f);
}

__device__ __forceinline__ void store_state(const Inst& in, const int64_t o, const State& s) {
  in.qc[o] = s.qc; in.nc[o] = s.nc; in.qr[o] = s.qr; in.nr[o] = s.nr;
  in.qi[o] = s.qi; in.qm[o] = s.qm; in.ni[o] = s.ni; in.bm[o] = s.bm;
  in.qv[o] = s.qv; in.th[o] = s.th;
}
__device__ __forceinline__ void load_state(const Inst& in, const int64_t o, State& s) {
  s.qc = in.qc[o]; s.nc = in.nc[o]; s.qr = in.qr[o]; s.nr = in.nr[o];
  s.qi = in.qi[o]; s.qm = in.qm[o]; s.ni = in.ni[o]; s.bm = in.bm[o];
  s.qv = in.qv[o]; s.th = in.th[o];
}

/* The species below their thresholds at the start of a level's part1: to
 * vapour (or, small ice above freezing, to rain), and the droplet number of a
 * level that keeps its cloud (`activated`).  A +0 moves nothing, so its FP64
 * updates are skipped (bitwise the same result).  Returns whether the potential
 * temperature changed. */
template <class F>
__device__ __forceinline__ bool part1_thresholds(State& s, double T, double inv_exner, double qvssi, F&& activated) {
  bool th_changed = false;
  if (dlt(s.qc, C::QSMALL)) {
    if (dnz(s.qc)) {
      s.qv = s.qv + s.qc;
      s.th = s.th - inv_exner * s.qc * C::LatVap * C::INV_CP;
      th_changed = true;
    }
    s.qc = 0;
    s.nc = 0;
  } else {
    s.nc = activated(s.nc);
  }
  if (dlt(s.qr, C::QSMALL)) {
    if (dnz(s.qr)) {
      s.qv = s.qv + s.qr;
      s.th = s.th - inv_exner * s.qr * C::LatVap * C::INV_CP;
      th_changed = true;
    }
    s.qr = 0;
    s.nr = 0;
  }
  if (dlt(s.qi, C::QSMALL) || (dlt(s.qi, 1.e-8) && dlt_neg(qvssi, -0.1))) {
    if (dnz(s.qi)) {
      s.qv = s.qv + s.qi;
      s.th = s.th - inv_exner * s.qi * (C::LatVap + C::LatIce) * C::INV_CP;
      th_changed = true;
    }
    s.qi = 0; s.ni = 0; s.qm = 0; s.bm = 0;
  }
  if (dge(s.qi, C::QSMALL) && dlt(s.qi, 1.e-8) && dge(T, C::T_zerodegc)) {
    s.qr = s.qr + s.qi;
    s.th = s.th - inv_exner * s.qi * C::LatIce * C::INV_CP;
    th_changed = true;
    s.qi = 0; s.ni = 0; s.qm = 0; s.bm = 0;
  }
  return th_changed;
}

/* Saturation, the rest of p3_main_part1 and p3_main_part2 of one level with a
 * hydrometeor in the FP32-bulk form (p3_main_part2_impl.hpp,
 * same order of processes).  The FP64 state is read once and shadowed in
 * FP32; the in-cloud values, DSDs, table lookups, process rates and limiter
 * ratios are FP32, while the thresholds test the FP64 state.  The vapour
 * residuals, the melting / wet-growth departures and the state update are
 * FP64.  A DSD or rime limiter that changes an in-cloud value rewrites the
 * FP64 state and its shadow. */
__device__ __forceinline__ void hydro_level_bulk(const Inst& in, const int col, const int k, const KParams<float>& kp,
                                                 const Tabs<float>& tb, const float dtf, const float inv_dtf,
                                                 bool& hydro, uint32_t& err) {
  const RuntimeDev& rt = kp.rt;
  const bool predictNc = in.predictNc != 0, prescribedCCN = in.prescribedCCN != 0;
  const bool do_ice = rt.do_ice_production != 0;
  const double inv_dt_d = f2d(inv_dtf);
  const int64_t o = int64_t(col) * in.ld + k;
  const float rho = scr_f(in, S_RHO, col)[k], rhofaci = scr_f(in, S_RHOFACI, col)[k], acn = scr_f(in, S_ACN, col)[k];
  double T = scr_at(in, S_TATM, col)[k];
  State s;
  load_state(in, o, s);
  const double inv_exner = in.inv_exner[o];
  const double cld_i = read_now(in.cld_frac_i + o), cld_l = read_now(in.cld_frac_l + o),
               cld_r = read_now(in.cld_frac_r + o);
  /* one Newton reciprocal of the pressure, times ep_2, shared by both
   * saturation ratios, the melting departure and the supersaturation limiter;
   * the supersaturation ratio (threshold and rate input) in FP32 */
  const double ep_inv_p = C::ep_2 * rcp_newton1(dmax_c(in.pres[o], 1.e-3));
  const double qvsi = __dmul_rn(svp_tabulated(rt.svp_tab, T, true, err), ep_inv_p);
  const double qvssi = f2d(float(s.qv) / float(qvsi) - 1.0f);
  const double qvsl = __dmul_rn(svp_tabulated(rt.svp_tab, T, false, err), ep_inv_p);
  if (part1_thresholds(s, T, inv_exner, qvssi, [&](double nc) {
        if (prescribedCCN) return vmax(nc, rt.spa_ccn_to_nc_factor * in.nccn[o] * in.cld_frac_l[o]);
        if (predictNc) return dmax0(nc + in.nc_nuceat_tend[o] * double(in.dt));
        return __dmul_rn(C::NCCNST, f2d(1.0f / rho));
      })) {
    T = __dmul_rn(s.th, rcp_newton1(inv_exner));
    scr_at(in, S_TATM, col)[k] = T;
  }
  if (dlt(s.qc, C::QSMALL) && dlt(s.qr, C::QSMALL) && dlt(s.qi, C::QSMALL)) {
    /* Without a hydrometeor left and where ice cannot nucleate (that needs
     * T < Tmelt - 15 and a supersaturation of 0.05; the test leaves a margin for
     * the float temperature) the level has no process rate: every tendency
     * output is the +0 of the first pass, except vap_liq_exchange = -(+0). */
    const bool dry_cold = dlt(T, C::T_zerodegc) && dlt_neg(qvssi, -0.05);
    if (dry_cold || ((predictNc || prescribedCCN) && !(dlt(T, C::Tmelt - 14.0) && dge(qvssi, 0.04)))) {
      if (!dry_cold) in.vap_liq_exchange[o] = -0.0;
      store_state(in, o, s);
      return;
    }
  }

  const float inv_rho = 1.0f / rho;
  const float T_r = float(T), qvsi_r = float(qvsi);
  const float cl = float(cld_l), ci = float(cld_i), cr = float(cld_r);
  const float icl = 1.0f / cl, ici = 1.0f / ci, icr = 1.0f / cr;
  /* FP32 shadows of the state (kept equal to float(s.x) where s.x changes) */
  /* part1 left a species below qsmall at zero */
  float qc0 = 0, nc0 = 0, qr0 = 0, nr0 = 0, qi0 = 0, ni0 = 0, qm0 = 0, bm0 = 0;
  if (dnz(s.qc) || dnz(s.nc)) {
    qc0 = float(s.qc);
    nc0 = float(s.nc);
  }
  if (dnz(s.qr) || dnz(s.nr)) {
    qr0 = float(s.qr);
    nr0 = float(s.nr);
  }
  if (dnz(s.qi) || dnz(s.ni)) {
    qi0 = float(s.qi);
    ni0 = float(s.ni);
  }
  if (dnz(s.qm) || dnz(s.bm)) {
    qm0 = float(s.qm);
    bm0 = float(s.bm);
  }
  constexpr float QS = float(C::QSMALL);

  /* calculate_incloud_mixingratios (bm uses 1/cld_frac_l, p3_incloud_mixingratios_impl.hpp:49) */
  float qc_in = 0, nc_in = 0, qr_in = 0, nr_in = 0, qi_in = 0, ni_in = 0, qm_in = 0, bm_in = 0;
  if (dge(s.qc, C::QSMALL)) { qc_in = qc0 * icl; nc_in = vmax(nc0 * icl, 0.0f); }
  if (dge(s.qi, C::QSMALL)) { qi_in = qi0 * ici; ni_in = vmax(ni0 * ici, 0.0f); }
  if (dge(s.qi, C::QSMALL) && dge(s.qm, C::QSMALL)) { qm_in = qm0 * ici; bm_in = vmax(bm0 * icl, 0.0f); }
  if (dge(s.qr, C::QSMALL)) { qr_in = qr0 * icr; nr_in = vmax(nr0 * icr, 0.0f); }
  {
    constexpr float il = float(C::incloud_limit), pl = float(C::precip_limit);
    if (qc_in > il || qi_in > il || qr_in > pl || bm_in > il) {
      qc_in = vmin(qc_in, il);
      qi_in = vmin(qi_in, il);
      bm_in = vmin(bm_in, il);
      qr_in = vmin(qr_in, pl);
    }
  }

  Rates<float> r;
  r.zero();
  PhysVars<float> v;
  v.mu = v.dv = v.sc = v.dqsdt = v.dqsidt = v.ab = v.abi = v.kap = v.eii = 0.0f;
  float tv_fallspd = 0, tv_selfcol = 0, tv_qc2qi = 0, tv_melt = 0, tv_nr = 0, tv_qr2qi = 0, tv_lammax = 0,
        tv_lammin = 0, tv_vent = 0;
  float mu_c = 0, lamc = 0, mu_r = 0, lamr = 0, cdistr = 0, logn0r = 0;
  float epsi = 0, epsr = 0, epsi_tot = 0;
  float rho_qm_cloud = 400.0f;
  bool wet = false;
  const auto rain_size = [&] { return m_cbrt(qr_in / (float(C::Pi) * float(C::RHO_H2O) * nr_in)); };

  if (qc_in >= QS || qr_in >= QS || qi_in >= QS) {
    get_time_space_phys_variables<float>(T_r, m_pow(T_r, 1.5f), m_pow(T_r, 1.81f), float(in.pres[o]), rho, float(qvsl), qvsi_r, v);
    {
      float n_out = nc_in;
      get_cloud_dsd2<float>(qc_in, n_out, mu_c, rho, lamc);
      if (n_out != nc_in) {
        nc_in = n_out;
        s.nc = f2d(n_out) * cld_l;
        nc0 = float(s.nc);
      }
    }
    {
      float n_out = nr_in;
      get_rain_dsd2<float>(qr_in, n_out, mu_r, lamr, rt);
      const bool changed = n_out != nr_in;
      nr_in = n_out;
      if (qr_in >= QS) {
        cdistr = nr_in / rt.f.g_mur1;
        logn0r = m_log10(cdistr) + (mu_r + 1.0f) * m_log10(lamr);
      }
      if (changed) {
        s.nr = f2d(n_out) * cld_r;
        nr0 = float(s.nr);
      }
    }
    impose_max_total_ni(ni_in, rt.f.max_total_ni, inv_rho);
    if (qi_in >= QS) {
      ni_in = vmax(ni_in, float(C::NSMALL));
      nr_in = vmax(nr_in, float(C::NSMALL));
      float qm_f = qm_in, bm_f = bm_in;
      const float rhop = calc_bulk_rho_rime<float>(qi_in, qm_f, bm_f, rt);
      if (qm_f != qm_in) {
        qm_in = qm_f;
        s.qm = f2d(qm_f) * cld_i;
        qm0 = float(s.qm);
      }
      if (bm_f != bm_in) {
        bm_in = bm_f;
        s.bm = f2d(bm_f) * cld_i;
        bm0 = float(s.bm);
      }
      TableIce<float> ti;
      lookup_ice<float>(qi_in, ni_in, qm_in, rhop, ti);
      TableRain<float> trn;
      lookup_rain<float>(qr_in, nr_in, trn, rain_size);
      float ta[4], tc[4];
      apply_table_ice4<float>(tb, ti, 0, ta); /* columns 0, 1, 6, 7 */
      apply_table_ice4<float>(tb, ti, 4, tc); /* columns 2, 3, 4, 9 */
      tv_fallspd = ta[1];
      tv_selfcol = tc[0];
      tv_qc2qi = tc[1];
      tv_melt = tc[2];
      tv_lammax = ta[2];
      tv_lammin = ta[3];
      tv_vent = tc[3];
      if (qr_in >= QS) {
        tv_nr = apply_table_coll<float>(0, tb, ti, trn);
        tv_qr2qi = apply_table_coll<float>(1, tb, ti, trn);
      }
      ni_in = vmin(ni_in, tv_lammax * ni_in);
      ni_in = vmax(ni_in, tv_lammin * ni_in);
    }
    const double dT0 = T - C::Tmelt;
    const double dqv0 = kp.esat0 * ep_inv_p - s.qv;
    const auto vent = [&] { return tv_melt + tv_vent * m_cbrt(v.sc) * m_sqrt(rhofaci * rho / v.mu); };
    const auto imm = [&] { return m_exp(rt.f.immersion_freezing_exponent * (float(C::T_zerodegc) - T_r)); };
    if (do_ice) {
      ice_cldliq_collection<float>(rho, T, rhofaci, tv_qc2qi, qi_in, qc_in, ni_in, nc_in, r, rt);
      ice_rain_collection<float>(rho, T, rhofaci, logn0r, tv_nr, tv_qr2qi, qi_in, ni_in, qr_in, r, rt);
      ice_self_collection<float>(rho, rhofaci, tv_selfcol, v.eii, qm_in, qi_in, ni_in, r);
    }
    ice_melting<float>(rho, dT0, dqv0, v, qi_in, ni_in, r, vent);
    if (do_ice) {
      wet = ice_cldliq_wet_growth<float>(rho, dT0, dqv0, v, qc_in, qi_in, ni_in, qr_in, r, vent);
    }
    /* ice_relaxation_timescale, p3_ice_relaxation_timescale_impl.hpp:9-37 */
    if (qi_in >= QS && dlt(T, C::Tmelt)) {
      epsi = ((tv_melt + tv_vent * m_cbrt(v.sc) * m_sqrt(rhofaci * rho / v.mu)) * 2.0f * float(C::Pi) * rho *
              v.dv) * ni_in;
      epsi_tot = epsi_tot + epsi;
    }
    rho_qm_cloud = calc_rime_density<float>(T_r, rhofaci, tv_fallspd, acn, lamc, mu_c, qc_in,
                                            r.qc2qi_collect_tend);
    if (do_ice) {
      cldliq_immersion_freezing<float>(T_r, lamc, mu_c, nc_in, qc_in, r, rt, imm);
      rain_immersion_freezing<float>(T_r, lamr, mu_r, cdistr, qr_in, r, rt, imm);
    }
    /* calc_liq_relaxation_timescale, p3_calc_liq_relaxation_timescale_impl.hpp:13-43 */
    if (qr_in >= QS) {
      Table3<float> t3;
      lookup3<float>(mu_r, lamr, rt, t3);
      epsr = 2.0f * float(C::Pi) * cdistr * rho * v.dv *
             (float(C::f1r) * rt.f.g_mur2 / lamr +
              float(C::f2r) * m_sqrt(rho / v.mu) * m_cbrt(v.sc) * apply_table3<float>(tb, tb.revap, t3));
    }
    evaporate_rain_bulk(qr_in, qc_in, nr_in, qi_in, cl, cr, s.qv, in.qv_prev[o], qvsl, qvsi, v.ab, v.abi, epsr,
                        epsi_tot, T, in.t_prev[o], v.dqsdt, dtf, inv_dtf, inv_dt_d, r.qr2qv_evap_tend,
                        r.nr_evap_tend);
    if (do_ice) {
      ice_deposition_sublimation_bulk(qi_in, ni_in, T, qvsl, qvsi, epsi, v.abi, s.qv, inv_dtf, r.qv2qi_vapdep_tend,
                                      r.qi2qv_sublim_tend, r.ni_sublim_tend, r.qc2qi_berg_tend);
    }
  }
  if (do_ice) {
    ice_nucleation<float>(T_r, inv_rho, ni0, float(in.ni_activated[o]), qvssi, inv_dtf, predictNc, prescribedCCN,
                          r, rt);
  }
  cloud_water_autoconversion<float>(rho, qc_in, nc_in, r, rt);
  if (qc_in >= QS) r.nc_selfcollect_tend = 0.0f;
  cloud_rain_accretion<float>(qc_in, nc_in, qr_in, r, rt);
  rain_self_collection<float>(rho, qr_in, nr_in, r, rt, rain_size);
  back_to_cell_average<float>(cl, cr, ci, r);

  /* limiters on the FP32 rates (FP64 vapour residuals), one FP64
   * application of each prognostic's FP32 tendency */
  const int wlim = water_conservation<float>(qc0, qr0, qi0, dtf, r);
  const int nlim = number_conservation<float>(nc0, nr0, ni0, dtf, r);
  const Rates<float> r_lim = r;
  ice_supersat_conservation_bulk(r, cld_i, s.qv, qvsi, qvsi_r, T_r, dtf);
  prevent_liq_supersaturation_bulk(ep_inv_p, T, s.qv, dtf, r, rt, err);
  update_prognostics_bulk(r, inv_exner, predictNc, prescribedCCN, wet, dtf, rho_qm_cloud, f2d(inv_rho), wlim, nlim,
                          r_lim, qi0, qm0, bm0, s);

  in.qv2qi_depos_tend[o] = f2d_zero(r.qv2qi_vapdep_tend - r.qi2qv_sublim_tend + r.qv2qi_nucleat_tend);
  in.precip_total_tend[o] = f2d_zero(r.qc2qr_accret_tend + r.qc2qr_autoconv_tend + r.qc2qr_ice_shed_tend +
                                r.qc2qi_collect_tend);
  in.nevapr[o] = f2d_zero(r.qi2qv_sublim_tend + r.qr2qv_evap_tend);
  in.vap_ice_exchange[o] = f2d_zero(r.qv2qi_vapdep_tend - r.qi2qv_sublim_tend + r.qv2qi_nucleat_tend);
  in.vap_liq_exchange[o] = f2d_zero(-r.qr2qv_evap_tend);
  in.liq_ice_exchange[o] = f2d_zero(r.qc2qi_hetero_freeze_tend + r.qr2qi_immers_freeze_tend - r.qi2qr_melt_tend +
                               r.qc2qi_berg_tend + r.qc2qi_collect_tend + r.qr2qi_collect_tend);

  hydro |= clip_to_vapour(s, inv_exner);
  if (dge(s.ni, 1e-20)) {
    /* impose_max_total_ni as a factor applied only when it limits */
    const float f = vmin(rt.f.max_total_ni * inv_rho * ci / float(s.ni), 1.0f);
    if (f < 1.0f) s.ni = s.ni * f2d(f);
  }
  store_state(in, o, s);
}

/* Saturation over ice and p3_main_part2 of one level without hydrometeors in
 * the FP32-bulk form, where ice nucleation is the only process that can have a
 * rate: the same operations that hydro_level_bulk leaves once every other rate
 * is +0 (a fifth of its FP64 instructions, which it spends on converting and
 * updating a state of zeros). */
__device__ __forceinline__ void nucleation_level_bulk(const Inst& in, const int col, const int k,
                                                      const KParams<float>& kp, const float dtf, const float inv_dtf,
                                                      bool& hydro, uint32_t& err) {
  const RuntimeDev& rt = kp.rt;
  const bool predictNc = in.predictNc != 0, prescribedCCN = in.prescribedCCN != 0;
  const int64_t o = int64_t(col) * in.ld + k;
  const double T = scr_at(in, S_TATM, col)[k];
  State s;
  s.qc = s.nc = s.qr = s.nr = s.qm = s.bm = 0.0;
  /* all reads at once (345,600 x 128 5.28 -> 5.15 ms) */
  s.qv = read_now(in.qv + o);
  s.th = read_now(in.th + o);
  const double cld_i = read_now(in.cld_frac_i + o), inv_exner = read_now(in.inv_exner + o);
  const float rho = read_now(scr_f(in, S_RHO, col) + k);
  const double ep_inv_p = C::ep_2 * rcp_newton1(dmax_c(in.pres[o], 1.e-3));
  const double qvsi = __dmul_rn(svp_tabulated(rt.svp_tab, T, true, err), ep_inv_p);
  const double qvssi = f2d(float(s.qv) / float(qvsi) - 1.0f);
  if (!(dlt(T, C::Tmelt - 14.0) && dge(qvssi, 0.04))) return;
  const float T_r = float(T), inv_rho = 1.0f / rho;
  const float activated = (predictNc && !prescribedCCN) ? float(in.ni_activated[o]) : 0.0f; /* read in that case only */
  Rates<float> r;
  r.zero();
  ice_nucleation<float>(T_r, inv_rho, 0.0f, activated, qvssi, inv_dtf, predictNc, prescribedCCN, r, rt);
  if (r.ni_nucleat_tend == 0.0f && r.qv2qi_nucleat_tend == 0.0f) return;
  ice_supersat_conservation_bulk(r, cld_i, s.qv, qvsi, float(qvsi), T_r, dtf);
  const float dni = r.ni_nucleat_tend * dtf;
  s.qi = f2d(r.qv2qi_nucleat_tend * dtf);
  s.ni = f2d(dni);
  s.qv = s.qv - s.qi;
  s.th = s.th + inv_exner * (((C::LatVap + C::LatIce) * C::INV_CP) * s.qi);
  const double depos = f2d(r.qv2qi_nucleat_tend);
  in.qv2qi_depos_tend[o] = depos;
  in.vap_ice_exchange[o] = depos;
  hydro |= clip_to_vapour(s, inv_exner);
  if (dge(s.ni, 1e-20)) {
    const float f = vmin(rt.f.max_total_ni * inv_rho * float(cld_i) / dni, 1.0f);
    if (f < 1.0f) s.ni = s.ni * f2d(f);
  }
  in.qi[o] = s.qi;
  in.ni[o] = s.ni;
  in.qv[o] = s.qv;
  in.th[o] = s.th;
}

/* ------------------------------------------------------------------ */
/* one column                                                          */
/* ------------------------------------------------------------------ */
/* Saturation vapour pressure (murphy_koop_svp) of the FP64 part1+2 with the
 * logarithm of the temperature shared by its liquid and ice forms. */
__device__ __forceinline__ double svp_liquid(double t, double logt) {
  return m_exp(54.842763 - m_div(6763.22, t) - (4.210 * logt) + (0.000367 * t) +
               (m_tanh(0.0415 * (t - 218.8)) * (53.878 - m_div(1331.22, t) - (9.44523 * logt) + 0.014025 * t)));
}
__device__ __forceinline__ double svp_ice(double t, double logt) {
  return m_exp(9.550426 - m_div(5723.265, t) + (3.53068 * logt) - (0.00728332 * t));
}
__device__ __forceinline__ void saturation_f64(const double T, const double pres, double& qvsl, double& qvsi) {
  const double p = vmax(pres, 1.e-3);
  const double logt = m_log(T);
  qvsl = m_div(C::ep_2 * svp_liquid(T, logt), p);
  qvsi = T < C::Tmelt ? m_div(C::ep_2 * svp_ice(T, logt), p) : qvsl;
}
/* What a CTA that works on one column forms of a hydrometeor level ahead, in
 * shared memory, a warp per job: its time is the latency of one level's chain of
 * library functions (a pow 5,700 cycles), and the other warps have nothing to do.
 * One column of 72 levels 89 -> 80 us, 64 x 72 96 -> 88 us; the same bits. */
enum { kPreT15 = 0, kPreT181, kPreRhofaci, kPreQvsl, kPreQvsi, kPreFields };
constexpr int kPreLevels = 512; /* shallower columns only: 40 B of shared memory a level */
__device__ __forceinline__ void level_ahead_f64(const Inst& in, const int col, const int k, const int job,
                                                double* pre, const int stride) {
  const double T = scr_at(in, S_TATM, col)[k];
  if (job == 0) {
    pre[kPreT15 * stride] = m_pow(T, 1.5);
  } else if (job == 1) {
    pre[kPreT181 * stride] = m_pow(T, 1.81);
  } else if (job == 2) {
    pre[kPreRhofaci * stride] = m_pow(C::RHO_600MB * m_div(1.0, scr_at(in, S_RHO, col)[k]), .54);
  } else {
    saturation_f64(T, in.pres[int64_t(col) * in.ld + k], pre[kPreQvsl * stride], pre[kPreQvsi * stride]);
  }
}

/* Saturation, the rest of p3_main_part1 and p3_main_part2 of one level with a
 * hydrometeor in the FP64 form (p3_main_part2_impl.hpp, same order of
 * processes).  Each library function (a pow holds the FP64 pipe for 1,500
 * cycles) is evaluated once and only where a process reads it: the cube root of
 * the Schmidt number and the ventilation term serve melting, wet growth,
 * relaxation and rain evaporation; the viscosity terms need rain or ice, rhofaci
 * ice, acn cloud and ice, and logn0r rain and ice. */
__device__ __forceinline__ void hydro_level_f64(const Inst& in, const int col, const int k, const KParams<double>& kp,
                                                const Tabs<double>& tb, const double dt, const double inv_dt,
                                                bool& hydro, uint32_t& err, const double* pre = nullptr,
                                                const int pre_stride = 0) {
  const RuntimeDev& rt = kp.rt;
  const bool predictNc = in.predictNc != 0, prescribedCCN = in.prescribedCCN != 0;
  const bool do_ice = rt.do_ice_production != 0;
  const int64_t o = int64_t(col) * in.ld + k;
  const double rho = scr_at(in, S_RHO, col)[k];
  double T = scr_at(in, S_TATM, col)[k];
  State s;
  load_state(in, o, s);
  const double inv_exner = in.inv_exner[o];
  const double pres = in.pres[o];
  double qvsl, qvsi;
  if (pre) {
    qvsl = pre[kPreQvsl * pre_stride];
    qvsi = pre[kPreQvsi * pre_stride];
  } else {
    saturation_f64(T, pres, qvsl, qvsi);
  }
  const double qvssi = m_div(s.qv, qvsi) - 1;
  const double T_before = T;
  const bool th_changed = part1_thresholds(s, T, inv_exner, qvssi, [&](double nc) {
    if (prescribedCCN)
      return vmax(nc, m_div(rt.spa_ccn_to_nc_factor * in.nccn[o], m_div(1.0, in.cld_frac_l[o])));
    if (predictNc) return dmax0(nc + in.nc_nuceat_tend[o] * dt);
    return __dmul_rn(C::NCCNST, m_div(1.0, rho));
  });
  if (th_changed) {
    T = __dmul_rn(s.th, m_div(1.0, inv_exner));
    scr_at(in, S_TATM, col)[k] = T;
  }
  if (dlt(s.qc, C::QSMALL) && dlt(s.qr, C::QSMALL) && dlt(s.qi, C::QSMALL) && dlt(T, C::T_zerodegc) &&
      dlt_neg(qvssi, -0.05)) {
    store_state(in, o, s);
    return;
  }

  const double cld_i = in.cld_frac_i[o], cld_l = in.cld_frac_l[o], cld_r = in.cld_frac_r[o];
  const double inv_rho = m_div(1.0, rho);
  Incld inc;
  calc_incloud(s.qc, s.qr, s.qi, s.qm, s.nc, s.nr, s.ni, s.bm, m_div(1.0, cld_l), m_div(1.0, cld_i),
               m_div(1.0, cld_r), inc);

  Rates<double> r;
  r.zero();
  PhysVars<double> v;
  v.mu = v.dv = v.sc = v.dqsdt = v.dqsidt = v.ab = v.abi = v.kap = v.eii = 0.0;
  double tv_fallspd = 0, tv_selfcol = 0, tv_qc2qi = 0, tv_melt = 0, tv_nr = 0, tv_qr2qi = 0, tv_lammax = 0,
         tv_lammin = 0, tv_vent = 0;
  double mu_c = 0, lamc = 0, mu_r = 0, lamr = 0, cdistr = 0, logn0r = 0;
  double epsi = 0, epsr = 0, epsi_tot = 0;
  double rho_qm_cloud = 400.0;
  double rain_size = 0; /* (qr / (pi rho_w nr))^(1/3) */
  bool wet = false;

  const bool has_c = dge(inc.qc, C::QSMALL), has_r = dge(inc.qr, C::QSMALL), has_i = dge(inc.qi, C::QSMALL);
  if (has_c || has_r || has_i) {
    double cbrt_sc = 0;
    if (has_r || has_i) {
      const bool known = pre && !th_changed;
      get_time_space_phys_variables<double>(T, known ? pre[kPreT15 * pre_stride] : m_pow(T, 1.5),
                                            known ? pre[kPreT181 * pre_stride] : m_pow(T, 1.81), pres, rho, qvsl, qvsi,
                                            v);
      cbrt_sc = m_cbrt(v.sc);
    }
    {
      const double n_in = inc.nc;
      double n_out = n_in;
      get_cloud_dsd2<double>(inc.qc, n_out, mu_c, rho, lamc);
      apply_n_adjust(inc.nc, n_in, n_out);
      s.nc = inc.nc * cld_l;
    }
    {
      const double n_in = inc.nr;
      double n_out = n_in;
      get_rain_dsd2<double>(inc.qr, n_out, mu_r, lamr, rt);
      apply_n_adjust(inc.nr, n_in, n_out);
      if (has_r) {
        cdistr = m_div(inc.nr, rt.g_mur1);
        if (has_i) logn0r = m_log10(cdistr) + (mu_r + 1.0) * m_log10(lamr);
      }
      s.nr = inc.nr * cld_r;
    }
    impose_max_total_ni(inc.ni, rt.max_total_ni, inv_rho);
    if (has_i) {
      inc.ni = dmax_c(inc.ni, C::NSMALL);
      inc.nr = dmax_c(inc.nr, C::NSMALL);
    }
    if (has_r) rain_size = m_cbrt(m_div(inc.qr, C::Pi * C::RHO_H2O * inc.nr));
    double rhofaci = 0, vent = 0;
    if (has_i) {
      rhofaci = pre ? pre[kPreRhofaci * pre_stride] : m_pow(C::RHO_600MB * inv_rho, .54);
      const double rhop = calc_bulk_rho_rime(inc.qi, inc.qm, inc.bm, rt);
      s.qm = inc.qm * cld_i;
      s.bm = inc.bm * cld_i;
      TableIce<double> ti;
      lookup_ice<double>(inc.qi, inc.ni, inc.qm, rhop, ti);
      TableRain<double> trn;
      lookup_rain<double>(inc.qr, inc.nr, trn, [&] { return rain_size; });
      double ta[4], tc[4];
      apply_table_ice4<double>(tb, ti, 0, ta); /* columns 0, 1, 6, 7 */
      apply_table_ice4<double>(tb, ti, 4, tc); /* columns 2, 3, 4, 9 */
      tv_fallspd = ta[1];
      tv_selfcol = tc[0];
      tv_qc2qi = tc[1];
      tv_melt = tc[2];
      tv_lammax = ta[2];
      tv_lammin = ta[3];
      tv_vent = tc[3];
      if (has_r) {
        tv_nr = apply_table_coll<double>(0, tb, ti, trn);
        tv_qr2qi = apply_table_coll<double>(1, tb, ti, trn);
      }
      inc.ni = vmin(inc.ni, tv_lammax * inc.ni);
      inc.ni = vmax(inc.ni, tv_lammin * inc.ni);
      vent = tv_melt + tv_vent * cbrt_sc * m_sqrt(m_div(rhofaci * rho, v.mu));
    }
    const double qi_r = inc.qi, qc_r = inc.qc, ni_r = inc.ni, nc_r = inc.nc, qr_r = inc.qr;
    const double dT0 = T - C::Tmelt;
    const double dqv0 = m_div(C::ep_2 * kp.esat0, vmax(pres, 1.e-3)) - s.qv;
    if (do_ice) {
      ice_cldliq_collection<double>(rho, T, rhofaci, tv_qc2qi, qi_r, qc_r, ni_r, nc_r, r, rt);
      ice_rain_collection<double>(rho, T, rhofaci, logn0r, tv_nr, tv_qr2qi, qi_r, ni_r, qr_r, r, rt);
      ice_self_collection<double>(rho, rhofaci, tv_selfcol, v.eii, inc.qm, qi_r, ni_r, r);
    }
    ice_melting<double>(rho, dT0, dqv0, v, qi_r, ni_r, r, [&] { return vent; });
    if (do_ice) wet = ice_cldliq_wet_growth<double>(rho, dT0, dqv0, v, qc_r, qi_r, ni_r, qr_r, r, [&] { return vent; });
    /* ice_relaxation_timescale, p3_ice_relaxation_timescale_impl.hpp:9-37 */
    if (has_i && dlt(T, C::Tmelt)) {
      epsi = (vent * 2.0 * C::Pi * rho * v.dv) * ni_r;
      epsi_tot = epsi_tot + epsi;
    }
    if (has_c && has_i) {
      /* acn is that of the temperature before part1's changes, and v.mu that
       * viscosity wherever part1 changed none */
      const double dum = th_changed ? m_div(1.496e-6 * m_pow(T_before, 1.5), T_before + 120.0) : v.mu;
      const double acn = m_div(C::gravit * C::RHO_H2O, 18.0 * dum);
      rho_qm_cloud = calc_rime_density<double>(T, rhofaci, tv_fallspd, acn, lamc, mu_c, qc_r, r.qc2qi_collect_tend);
    }
    if (do_ice && (has_c || has_r) && T <= C::T_rainfrz) {
      const double e = m_exp(rt.immersion_freezing_exponent * (C::T_zerodegc - T));
      cldliq_immersion_freezing<double>(T, lamc, mu_c, nc_r, qc_r, r, rt, [&] { return e; });
      rain_immersion_freezing<double>(T, lamr, mu_r, cdistr, qr_r, r, rt, [&] { return e; });
    }
    /* calc_liq_relaxation_timescale, p3_calc_liq_relaxation_timescale_impl.hpp:13-43 */
    if (has_r) {
      Table3<double> t3;
      lookup3<double>(mu_r, lamr, rt, t3);
      epsr = 2.0 * C::Pi * cdistr * rho * v.dv *
             (m_div(C::f1r * rt.g_mur2, lamr) +
              C::f2r * m_sqrt(m_div(rho, v.mu)) * cbrt_sc * apply_table3<double>(tb, tb.revap, t3));
    }
    evaporate_rain(inc.qr, inc.qc, inc.nr, inc.qi, cld_l, cld_r, s.qv, in.qv_prev[o], qvsl, qvsi, v.ab, v.abi, epsr,
                   epsi_tot, T, in.t_prev[o], v.dqsdt, dt, r.qr2qv_evap_tend, r.nr_evap_tend);
    if (do_ice) {
      ice_deposition_sublimation(inc.qi, inc.ni, T, qvsl, qvsi, epsi, v.abi, s.qv, inv_dt, r.qv2qi_vapdep_tend,
                                 r.qi2qv_sublim_tend, r.ni_sublim_tend, r.qc2qi_berg_tend);
    }
  }
  if (do_ice) {
    ice_nucleation<double>(T, inv_rho, s.ni, in.ni_activated[o], qvssi, inv_dt, predictNc, prescribedCCN, r, rt);
  }
  cloud_water_autoconversion<double>(rho, inc.qc, inc.nc, r, rt);
  if (has_c) r.nc_selfcollect_tend = 0.0;
  cloud_rain_accretion<double>(inc.qc, inc.nc, inc.qr, r, rt);
  rain_self_collection<double>(rho, inc.qr, inc.nr, r, rt, [&] { return rain_size; });
  back_to_cell_average<double>(cld_l, cld_r, cld_i, r);

  water_conservation<double>(s.qc, s.qr, s.qi, dt, r);
  number_conservation<double>(s.nc, s.nr, s.ni, dt, r);
  ice_supersat_conservation(r, cld_i, s.qv, qvsi, m_div(s.th, inv_exner), dt);
  prevent_liq_supersaturation(pres, T, s.qv, dt, r, err);
  update_prognostics(r, inv_exner, predictNc, prescribedCCN, wet, dt, rho_qm_cloud, inv_rho, s);

  in.qv2qi_depos_tend[o] = r.qv2qi_vapdep_tend - r.qi2qv_sublim_tend + r.qv2qi_nucleat_tend;
  in.precip_total_tend[o] = r.qc2qr_accret_tend + r.qc2qr_autoconv_tend + r.qc2qr_ice_shed_tend + r.qc2qi_collect_tend;
  in.nevapr[o] = r.qi2qv_sublim_tend + r.qr2qv_evap_tend;
  in.vap_ice_exchange[o] = r.qv2qi_vapdep_tend - r.qi2qv_sublim_tend + r.qv2qi_nucleat_tend;
  in.vap_liq_exchange[o] = -r.qr2qv_evap_tend;
  in.liq_ice_exchange[o] = r.qc2qi_hetero_freeze_tend + r.qr2qi_immers_freeze_tend - r.qi2qr_melt_tend +
                           r.qc2qi_berg_tend + r.qc2qi_collect_tend + r.qr2qi_collect_tend;

  hydro |= clip_to_vapour(s, inv_exner);
  double ni_incld = m_div(s.ni, cld_i);
  impose_max_total_ni(ni_incld, rt.max_total_ni, inv_rho);
  s.ni = ni_incld * cld_i;
  store_state(in, o, s);
}

/* Saturation over ice and p3_main_part2 of one level without hydrometeors,
 * where ice nucleation is the only process that can have a rate: the same
 * operations that hydro_level_f64 leaves once every other rate is +0 (its
 * limiters do not engage, its sums add zeros). */
__device__ __forceinline__ void nucleation_level_f64(const Inst& in, const int col, const int k,
                                                     const KParams<double>& kp, const double dt, const double inv_dt,
                                                     bool& hydro) {
  const RuntimeDev& rt = kp.rt;
  const int64_t o = int64_t(col) * in.ld + k;
  const double T = scr_at(in, S_TATM, col)[k];
  State s;
  s.qc = s.nc = s.qr = s.nr = s.qm = s.bm = 0.0;
  s.qv = in.qv[o];
  const double qvsi = m_div(C::ep_2 * svp_ice(T, m_log(T)), vmax(in.pres[o], 1.e-3));
  const double qvssi = m_div(s.qv, qvsi) - 1;
  const double inv_rho = m_div(1.0, scr_at(in, S_RHO, col)[k]);
  Rates<double> r;
  r.zero();
  ice_nucleation<double>(T, inv_rho, 0.0, in.ni_activated[o], qvssi, inv_dt, in.predictNc != 0, in.prescribedCCN != 0,
                         r, rt);
  if (!dnz(r.ni_nucleat_tend) && !dnz(r.qv2qi_nucleat_tend)) return;
  s.th = in.th[o];
  const double cld_i = in.cld_frac_i[o], inv_exner = in.inv_exner[o];
  ice_supersat_conservation(r, cld_i, s.qv, qvsi, m_div(s.th, inv_exner), dt);
  const double q = r.qv2qi_nucleat_tend;
  s.qi = q * dt;
  s.ni = r.ni_nucleat_tend * dt;
  s.qv = fma(-q, dt, s.qv);
  s.th = fma(inv_exner * (q * (C::LatVap + C::LatIce) * C::INV_CP), dt, s.th);
  in.qv2qi_depos_tend[o] = q;
  in.vap_ice_exchange[o] = q;
  hydro |= clip_to_vapour(s, inv_exner);
  double ni_incld = m_div(s.ni, cld_i);
  impose_max_total_ni(ni_incld, rt.max_total_ni, inv_rho);
  in.qi[o] = s.qi;
  in.ni[o] = ni_incld * cld_i;
  in.qv[o] = s.qv;
  in.th[o] = s.th;
}

/* K1 of `ncol` neighbouring columns of one instance: p3_main_init,
 * p3_main_part1, p3_main_part2.  By one warp, or (WIDE) of one column by a CTA,
 * whose warps share the levels of the first pass and then take the lists 32
 * entries at a time.
 *
 * What bounds it: the FP64 pipe; in the FP64 form through the library functions
 * (pow 1,499 cycles of an SM, log 516, tanh 429, exp 274), whose bits ice
 * sedimentation carries into every later result, so they stay the library's; in
 * the FP32-bulk form through the state, residuals, saturation table and
 * conversions.  A first pass over all levels does what part1 does without
 * saturation (in the FP64 form the fall-speed factors, which only sedimentation
 * reads from here, are in fixed point), writes the hand-over rows and sorts the
 * levels into three classes:
 *   - with a hydrometeor: saturation, the rest of part1 and part2, on a list,
 *     so that a warp's lanes hold 32 such levels and not the few of them among
 *     32 consecutive ones;
 *   - without, cold, where the FP32 supersaturation over ice does not exclude
 *     nucleation: saturation over ice and nucleation, on a second list;
 *   - the rest: no process has a rate there.
 * The lists run over the pool of columns: a column's cloud fills a fraction of
 * a warp (18 of 128 levels in a cloud of 1-4 km), and the FP64 pipe takes
 * as long for one lane as for 32.  The same bits as with lists per column, where
 * part1's remainder and part2 were separate passes over arrays in shared memory
 * (FP64 16 lanes, FP32-bulk 32 lanes per column): 21,600 x 128 FP64 3.41 -> 2.36
 * ms, FP32-bulk 0.468 -> 0.33; 345,600 x 128 FP32-bulk 8.43 -> 4.86 ms; 1,537 x
 * 97 FP64 272 -> 239 us. */
template <class TR, bool WIDE>
__device__ void p3_part12(const Inst& in, const int col0, const int ncol, const KParams<TR>& kp, const Tabs<TR>& tb,
                          uint16_t* __restrict__ list, PoolScratch* __restrict__ ps, uint32_t& err) {
  constexpr bool kBulk = sizeof(TR) == sizeof(float);
  const RuntimeDev& rt = kp.rt;
  const unsigned lane = threadIdx.x & 31u;
  const int tid = WIDE ? int(threadIdx.x) : int(lane), step = WIDE ? int(blockDim.x) : 32;
  const int nk = in.nlev;
  const int total = ncol * nk;
  const double dt = in.dt;
  const bool do_ice = rt.do_ice_production != 0;
  int n_hyd = 0, n_nuc = 0;
  const unsigned below = (1u << lane) - 1u;
  if constexpr (WIDE) {
    __syncthreads(); /* every thread is done with the last column's lists */
    if (tid == 0) ps->n_hyd = ps->n_nuc = ps->active = 0;
    __syncthreads();
  } else {
    __syncwarp(); /* every lane is done with the last pool's lists */
  }

  /* ---------------- p3_main_init, part1 without saturation ---------------- */
  int c = 0, k = tid;
  for (int base = 0; base < total; base += step) {
    while (k >= nk && c < ncol) {
      k -= nk;
      ++c;
    }
    bool is_hyd = false, is_nuc = false;
    if (c < ncol) {
      const int col = col0 + c;
      const int64_t o = int64_t(col) * in.ld + k;
      const double inv_exner = in.inv_exner[o];
      double th = in.th[o];
      const double dz = in.dz[o];
      const double qv_in = in.qv[o];
      double qv = dmax0(qv_in);
      const double dpres = in.dpres[o];
      const double qc = in.qc[o], qr = in.qr[o], qi = in.qi[o];

      in.diag_eff_radius_qc[o] = 10.e-6;
      in.diag_eff_radius_qi[o] = 25.e-6;
      in.diag_eff_radius_qr[o] = 500.e-6;
      in.rho_qi[o] = 0;
      in.qv2qi_depos_tend[o] = 0;
      in.precip_total_tend[o] = 0;
      in.nevapr[o] = 0;
      in.liq_ice_exchange[o] = 0;
      in.vap_liq_exchange[o] = 0;
      in.vap_ice_exchange[o] = 0;

      double exner;
      if constexpr (kBulk) exner = rcp_newton1(inv_exner);
      else exner = m_div(1.0, inv_exner);
      double T = th * exner;
      if (dbits(T) <= 0 || dbits(T) > kInfBits) err |= kErrNumeric;
      if constexpr (kBulk) {
        /* rho and 1/rho only feed rates, fall speeds and fluxes (the
         * sedimentation's FP64 coefficient is g / dpres), so they are FP32 */
        const float rho_t = float(dpres) / (float(dz) * float(C::gravit));
        const float inv_rho_t = 1.0f / rho_t;
        const float tf = float(T);
        const float dum = float(1.496e-6) * m_pow(tf, float(1.5)) / (tf + float(120));
        scr_f(in, S_RHO, col)[k] = rho_t;
        scr_f(in, S_RHOFACR, col)[k] = m_pow(float(C::RHO_1000MB) * inv_rho_t, float(.54));
        scr_f(in, S_RHOFACI, col)[k] = m_pow(float(C::RHO_600MB) * inv_rho_t, float(.54));
        scr_f(in, S_ACN, col)[k] = float(C::gravit) * float(C::RHO_H2O) / (float(18) * dum);
      } else {
        const double rho = m_div(m_div(dpres, dz), C::gravit);
        const double inv_rho = m_div(1.0, rho);
        /* rhofaci is rhofacr times a constant */
        const double rhofacr = pow_fix(C::RHO_1000MB * inv_rho, .54);
        const double visc = m_div(1.496e-6 * (T * pow_fix(T, .5)), T + 120.0);
        scr_at(in, S_RHO, col)[k] = rho;
        scr_at(in, S_RHOFACR, col)[k] = rhofacr;
        scr_at(in, S_RHOFACI, col)[k] = rhofacr * kRhofaciOverR;
        scr_at(in, S_ACN, col)[k] = m_div(C::gravit * C::RHO_H2O, 18.0 * visc);
      }

      is_hyd = dge(qc, C::QSMALL) || dge(qr, C::QSMALL) || dge(qi, C::QSMALL);
      if (!is_hyd) {
        const bool traces = dnz(qc) || dnz(qr) || dnz(qi);
        if (do_ice && dlt(T, C::T_zerodegc))
          is_nuc = may_nucleate(T, float(T), float(qv), float(dmax_c(in.pres[o], 1.e-3)));
        /* nucleation is decided before a trace of condensate goes to vapour:
         * the general path does both */
        is_hyd = is_nuc && traces;
        is_nuc = is_nuc && !traces;
        if (!is_hyd) {
          if (traces) {
            /* a species below qsmall goes to vapour; a +0 moves nothing */
            if (dnz(qc)) {
              qv = qv + qc;
              th = th - inv_exner * qc * C::LatVap * C::INV_CP;
            }
            if (dnz(qr)) {
              qv = qv + qr;
              th = th - inv_exner * qr * C::LatVap * C::INV_CP;
            }
            if (dnz(qi)) {
              qv = qv + qi;
              th = th - inv_exner * qi * (C::LatVap + C::LatIce) * C::INV_CP;
            }
            T = th * exner;
            in.th[o] = th;
          }
          /* what was read and keeps its bits is not written back: this pass is
           * bound by its stores */
          if (dbits(qc)) in.qc[o] = 0;
          if (dbits(qr)) in.qr[o] = 0;
          if (dbits(qi)) in.qi[o] = 0;
          in.nc[o] = 0; in.nr[o] = 0; in.ni[o] = 0; in.qm[o] = 0; in.bm[o] = 0;
        }
      }
      if (dbits(qv) != dbits(qv_in)) in.qv[o] = qv;
      scr_at(in, S_TATM, col)[k] = T;
    }
    const unsigned b_hyd = __ballot_sync(0xffffffffu, is_hyd), b_nuc = __ballot_sync(0xffffffffu, is_nuc);
    const uint16_t entry = uint16_t((c << kPoolLevelBits) | k);
    if constexpr (WIDE) {
      if (lane == 0) {
        n_hyd = b_hyd ? int(atomicAdd(&ps->n_hyd, __popc(b_hyd))) : 0;
        n_nuc = b_nuc ? int(atomicAdd(&ps->n_nuc, __popc(b_nuc))) : 0;
      }
      n_hyd = __shfl_sync(0xffffffffu, n_hyd, 0);
      n_nuc = __shfl_sync(0xffffffffu, n_nuc, 0);
    }
    if (is_hyd) list[n_hyd + __popc(b_hyd & below)] = entry;
    if (is_nuc) list[total - 1 - n_nuc - __popc(b_nuc & below)] = entry;
    n_hyd += __popc(b_hyd);
    n_nuc += __popc(b_nuc);
    k += step;
  }
  for (c = 0; c < ncol; ++c) {
    const int64_t ci = int64_t(col0 + c) * in.ld_int;
    for (k = tid; k <= nk; k += step) {
      in.precip_liq_flux[ci + k] = 0;
      in.precip_ice_flux[ci + k] = 0;
    }
  }
  if (tid < ncol) {
    in.precip_liq_surf[col0 + tid] = 0;
    in.precip_ice_surf[col0 + tid] = 0;
  }
  /* the lists, and the rows other lanes wrote */
  if constexpr (WIDE) {
    __syncthreads();
    n_hyd = int(ps->n_hyd);
    n_nuc = int(ps->n_nuc);
  } else {
    __syncwarp();
  }

  /* ---------------- saturation, the rest of part1, part2 ---------------- */
  uint32_t active = 0; /* columns with a hydrometeor after part2 */
  /* a CTA's warps take one list or the other, a warp goes from the first to the second */
  const int n_pad = WIDE ? (n_hyd + 31) & ~31 : n_hyd;
  if constexpr (kBulk) {
    const float dtf = float(dt), inv_dtf = float(1 / dt);
    for (int j = tid; j < n_pad + n_nuc; j += step) {
      if (WIDE && j >= n_hyd && j < n_pad) continue;
      const int e = list[j < n_hyd ? j : total - 1 - (j - n_pad)];
      const int ce = e >> kPoolLevelBits, ke = e & ((1 << kPoolLevelBits) - 1);
      bool hydro = false;
      if (j < n_hyd) hydro_level_bulk(in, col0 + ce, ke, kp, tb, dtf, inv_dtf, hydro, err);
      else nucleation_level_bulk(in, col0 + ce, ke, kp, dtf, inv_dtf, hydro, err);
      active |= uint32_t(hydro) << ce;
    }
  } else {
    const double inv_dt = m_div(1.0, dt);
    double* const pre = WIDE && nk <= kPreLevels ? reinterpret_cast<double*>(list + pool_list_entries(1, nk)) : nullptr;
    if constexpr (WIDE) {
      if (pre) {
        /* four jobs a chunk of the list, a warp each */
        for (int u = tid >> 5; u < (n_pad >> 5) * 4; u += step >> 5) {
          const int j = (u >> 2) * 32 + int(lane);
          if (j < n_hyd) level_ahead_f64(in, col0, list[j] & ((1 << kPoolLevelBits) - 1), u & 3, pre + j, nk);
        }
        __syncthreads();
      }
    }
    for (int j = tid; j < n_pad + n_nuc; j += step) {
      if (WIDE && j >= n_hyd && j < n_pad) continue;
      const int e = list[j < n_hyd ? j : total - 1 - (j - n_pad)];
      const int ce = e >> kPoolLevelBits, ke = e & ((1 << kPoolLevelBits) - 1);
      bool hydro = false;
      if (j < n_hyd) hydro_level_f64(in, col0 + ce, ke, kp, tb, dt, inv_dt, hydro, err, WIDE && pre ? pre + j : nullptr, nk);
      else nucleation_level_f64(in, col0 + ce, ke, kp, dt, inv_dt, hydro);
      active |= uint32_t(hydro) << ce;
    }
  }
  active = __reduce_or_sync(0xffffffffu, active);
  if constexpr (WIDE) {
    if (lane == 0 && active) atomicOr(&ps->active, active);
    __syncthreads();
    if (tid == 0) in.cflag[col0] = int(ps->active);
  } else {
    if (int(lane) < ncol) in.cflag[col0 + lane] = (active >> lane) & 1u;
  }
}

/* K2 (FP64 form): cloud, rain and ice sedimentation of one column that went
 * on past part2.
 *
 * What bounds it: as the reference writes it (divisions, cbrt, log10 and the
 * table lerps in FP64) one ice level of one substep holds the FP64 pipe for
 * ~3,300 cycles of an SM and a rain level for ~1,400 (a warp instruction every
 * 16 cycles; a division takes 131, cbrt 227, log10 553).  Here the divisions,
 * the logarithm, the cube root and the table interpolation are 64-bit integer
 * arithmetic (16, 35, 73 and 42 cycles), the in-cloud values are never
 * formed (every quantity that the fall speeds need is a ratio of two fields of
 * one level, so the cloud fraction cancels; the in-cloud thresholds become
 * thresholds times the cloud fraction), and what stays FP64 is the flux:
 * one product, one difference and one multiply-add per field, with 1 / (dz rho)
 * formed once per level and V rho kept instead of V.  At 21,600 x 128: 15.8 ms
 * with integer divisions alone, 2.7 ms in this form (3.6 ms with exact 64-bit
 * high products, rounded quotients and 100 registers), 2.5 ms with the rime left
 * out where there is none; the FP64 pipe is 70 % busy then, the integer pipe 39 %.
 * The results differ from the reference's order of operations by rounding (1e-14
 * of a field's norm). */
template <class TR, int LANES, bool SPLIT = false>
__device__ void p3_sed(const Inst& in, const int col, const KParams<TR>& kp, const Tabs<TR>& tb,
                       double* __restrict__ sm, GroupScratch* gs, uint32_t& err) {
  static_assert(sizeof(TR) == sizeof(double), "the FP32-bulk sedimentation is p3_sed_bulk");
  if (in.cflag[col] == 0) return;
  const RuntimeDev& rt = kp.rt;
  const FixTables* const ft = &kFixTables;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & (LANES - 1);
  const int nk = in.nlev;
  const int S = kp.sm_stride;
  const int64_t co = int64_t(col) * in.ld;
  const int64_t ci = int64_t(col) * in.ld_int;
  const double dt = in.dt;
  const double inv_dt = m_div(1.0, dt);
  const bool predictNc = in.predictNc != 0;
  const int kbot = nk - 1;
  constexpr int kWarp = 32; /* lanes that shuffle with one another */
  double* const FR = sm + B_FR * S;   /* fall-speed factor of the species times rho */
  double* const CF = sm + B_CF * S;   /* 1 / (dz rho) */
  double* const QS = sm + B_QS * S;   /* QSMALL times the species' cloud fraction */
  double* const V1 = sm + B_V1 * S;   /* rho times the mass (V1) and number (V2) fall speed */
  double* const V2 = sm + B_V2 * S;
  double* const R0 = sm + B_R0 * S;   /* the species' fields */
  double* const R1 = sm + B_R1 * S;
  double* const R2 = sm + B_R2 * S;
  double* const R3 = sm + B_R3 * S;
  double* const PF = R2;              /* rain flux sum (rain has two fields) */
  const double* const rho_row = scr_at(in, S_RHO, col);

  /* Top and bottom of the three species (p3_find_impl.hpp) in one pass.  A
   * species only changes the levels from its top down to its final leading
   * edge; the others keep their values. */
  int top[3] = {1 << 30, 1 << 30, 1 << 30}, bot[3] = {-1, -1, -1};
  for (int k = lane; k < nk; k += LANES) {
    if (dge(in.qc[co + k], C::QSMALL)) { top[0] = min(top[0], k); bot[0] = k; }
    if (dge(in.qr[co + k], C::QSMALL)) { top[1] = min(top[1], k); bot[1] = k; }
    if (dge(in.qi[co + k], C::QSMALL)) { top[2] = min(top[2], k); bot[2] = k; }
  }
  if (LANES > 32 && lane < 3) gs->prt[lane] = 0;
  group_bounds<LANES, SPLIT>(mask, gs, top, bot);
  for (int k = min(top[0], min(top[1], top[2])) + lane; k < nk; k += LANES)
    CF[k] = ddiv_int(1.0, in.dz[co + k] * rho_row[k]);
  double precip_liq_surf = 0, precip_ice_surf = 0;

  auto species = [&](auto sp_tag) {
    constexpr int sp = decltype(sp_tag)::value;
    double* const g0 = sp == 0 ? in.qc : (sp == 1 ? in.qr : in.qi);
    double* const g1 = sp == 0 ? in.nc : (sp == 1 ? in.nr : in.ni);
    const double* const cldp = (sp == 0 ? in.cld_frac_l : (sp == 1 ? in.cld_frac_r : in.cld_frac_i)) + co;
    const double* const facp = scr_at(in, sp == 0 ? S_ACN : (sp == 1 ? S_RHOFACR : S_RHOFACI), col);
    const bool number = sp != 0 || predictNc; /* the number falls too */
    const int k_qxtop = top[sp];
    int k_qxbot = bot[sp];
    if (k_qxbot < 0) return; /* species absent (group-uniform) */

    for (int k = k_qxtop + lane; k < nk; k += LANES) {
      R0[k] = g0[co + k];
      R1[k] = g1[co + k];
      QS[k] = C::QSMALL * cldp[k];
      const double fac = sp == 2 ? rt.ice_sedimentation_factor * facp[k] : facp[k];
      FR[k] = fac * rho_row[k];
      if (sp == 2) {
        R2[k] = in.qm[co + k];
        R3[k] = in.bm[co + k];
      }
    }
    if (sp == 1) {
      for (int k = k_qxtop + lane; k <= nk; k += LANES) PF[k] = 0;
    }
    group_sync<LANES, SPLIT>(mask);

    /* From here on lane l owns levels k_qxtop + l + j*LANES in both the
     * fall-speed pass and the flux walk, so only shuffles cross lanes. */
    double dt_left = dt, prt_accum = 0.0;
    bool first = true;
    int nsub = 0;
    while (dgt(dt_left, C::dt_left_tol)) {
      if (++nsub > kMaxSubsteps) {
        err |= kErrSubstep;
        break;
      }
      /* fall speeds on [k_qxtop, k_qxbot] and the maximum of V / dz */
      double lmax = 0.0;
      for (int k = k_qxtop + lane; k <= k_qxbot; k += LANES) {
        const double qs = QS[k];
        double v1 = 0, v2 = 0;
        /* Ice without rime in the whole chunk: no rime density, and two table
         * corners instead of eight; below, its two fields' fluxes are left out as
         * well.  Nucleated ice over the clouds is most of the walk: 21,600 x 128
         * 2.66 -> 2.51 ms.  A warp of a wider group has one chunk and waits for the
         * others', so it does not look. */
        bool rime = true;
        if constexpr (sp == 2 && LANES == kWarp)
          rime = __any_sync(chunk_mask(k - lane, k_qxbot), dnz(R2[k]) || dnz(R3[k]));
        /* q: the mass field, limited in the first substep as the in-cloud
         * value is there; the field itself keeps its value */
        double q = R0[k], n = R1[k];
        bool present = dbits(q) > dbits(qs);
        if (first) {
          present = present && dge(q, C::QSMALL);
          if (present) {
            n = dmax0(n);
            /* incloud_limit and precip_limit over QSMALL */
            const double lim = qs * (sp == 1 ? C::precip_limit / C::QSMALL : C::incloud_limit / C::QSMALL);
            if (dbits(q) > dbits(lim)) q = lim;
          }
        }
        if (present) {
          if (dbits(n) < dbits(qs)) {
            const double least = qs * (C::NSMALL / C::QSMALL);
            if (dbits(n) < dbits(least)) n = least;
          }
          if (sp == 0) {
            /* get_cloud_dsd2 with in-cloud values, then the Stokes fall speeds
             * (p3_cloud_sed_impl.hpp:99-103) with Gamma(6+mu)/Gamma(4+mu) =
             * (5+mu)(4+mu) and Gamma(3+mu)/Gamma(1+mu) = (2+mu)(1+mu) */
            const double cld = cldp[k], n_in = m_div(n, cld);
            double mu_c, lamc, n_out = n_in;
            get_cloud_dsd2<double>(m_div(q, cld), n_out, mu_c, rho_row[k], lamc,
                                   [ft](double x) { return cbrt_fix(x, ft); });
            R1[k] = dbits(n_out) != dbits(n_in) ? n_out * cld : n;
            const double w = FR[k] * m_div(1.0, lamc * lamc);
            v1 = w * ((5.0 + mu_c) * (4.0 + mu_c));
            if (number) v2 = w * ((2.0 + mu_c) * (1.0 + mu_c));
          } else if (sp == 1) {
            if (rt.rain_fix) {
              const RainRow rr = rain_row(log2_of(raw_quotient(n, q), ft), rt.rain_kd, ft);
              if (rr.side != 0) n = (rr.side < 0 ? rt.rain_n_hi : rt.rain_n_lo) * q;
              const double4 t = kp.t3sed[(rt.t3_dumjj - 1) * kT3SedRows + rr.row - 1];
              v1 = fma(rr.frac, t.y, t.x);
              v2 = fma(rr.frac, t.w, t.z);
              if (dnz(rt.t3_wj)) {
                const double4 t1 = kp.t3sed[rt.t3_dumjj * kT3SedRows + rr.row - 1];
                v1 = fma(rt.t3_wj, fma(rr.frac, t1.y, t1.x) - v1, v1);
                v2 = fma(rt.t3_wj, fma(rr.frac, t1.w, t1.z) - v2, v2);
              }
              if (!(dbits(q) < kInfBits && dbits(n) < kInfBits)) v1 = d_from_bits(kNaNBits);
            } else {
              const double cld = cldp[k];
              double mu_r = 0, lamr, n_out = m_div(n, cld);
              get_rain_dsd2<double>(m_div(q, cld), n_out, mu_r, lamr, rt);
              Table3<double> t3;
              lookup3<double>(mu_r, lamr, rt, t3);
              v1 = apply_table3<double>(tb, tb.vm, t3);
              v2 = apply_table3<double>(tb, tb.vn, t3);
              n = n_out * cld;
            }
            v1 *= FR[k];
            v2 *= FR[k];
            R1[k] = n;
          } else {
            double m = R2[k], b = R3[k];
            int64_t hi, lo, vm, vn;
            int4 sh;
            const int64_t size = log2_of(raw_quotient(q, n), ft);
            if (rime) {
              if (first) {
                if (dge(m, C::QSMALL)) {
                  /* bm_incld uses 1 / cld_frac_l (p3_incloud_mixingratios_impl.hpp:49) */
                  b = dmax0(ddiv_int(b, in.cld_frac_l[co + k])) * cldp[k];
                  const double lim = qs * (C::incloud_limit / C::QSMALL);
                  if (dbits(b) > dbits(lim)) b = lim;
                } else {
                  m = 0;
                  b = 0;
                }
              }
              /* calc_bulk_rho_rime, p3/impl/p3_ice_sed_impl.hpp:14-64; the rime
               * density itself is only needed in fixed point */
              uint64_t rho52 = 0;
              const bool rimed = dbits(b) >= dbits(qs) || dbits(b) >= dbits(qs * (C::BSMALL / C::QSMALL));
              if (rimed && dbits(b) <= kInfBits) {
                const bool lt = dbits(m) < dbits(rt.min_rime_rho * b), gt = dbits(m) > dbits(rt.max_rime_rho * b);
                double rho_lim = lt ? rt.min_rime_rho : rt.max_rime_rho;
                if (!lt && !gt) {
                  rho52 = rho_q52(raw_quotient(m, b));
                  if (dbits(m) > dbits(q)) rho_lim = ddiv_int(m, b);
                } else {
                  rho52 = rho_q52(rho_lim);
                }
                const bool over = dbits(m) > dbits(q);
                if (over) m = q;
                if (lt || gt || over) b = ddiv_int(m, rho_lim);
              } else if (!rimed) {
                m = 0;
                b = 0;
              }
              if (dbits(m) < dbits(qs)) {
                m = 0;
                b = 0;
              }
              R2[k] = m;
              R3[k] = b;
              const IceCell cell = ice_cell_at(size, dnz(m) ? fix_of(raw_quotient(m, q), 60) : 0, rho52);
              const int64_t* const cf = kp.cell_sed + size_t(cell.cell) * (kCellCols * kCellCoefs);
              sh = __ldg(reinterpret_cast<const int4*>(kp.cell_sed_shift) + cell.cell);
              vn = ice_cell_value(cf, cell);
              vm = ice_cell_value(cf + kCellCoefs, cell);
              hi = ice_cell_value(cf + 2 * kCellCoefs, cell);
              lo = ice_cell_value(cf + 3 * kCellCoefs, cell);
            } else {
              const FixAxis a1 = ice_size_at(size);
              const int64_t* const cf = kp.cell_sed + size_t(a1.i) * (kCellCols * kCellCoefs);
              sh = __ldg(reinterpret_cast<const int4*>(kp.cell_sed_shift) + a1.i);
              vn = ice_cell_value_unrimed(cf, a1.w);
              vm = ice_cell_value_unrimed(cf + kCellCoefs, a1.w);
              hi = ice_cell_value_unrimed(cf + 2 * kCellCoefs, a1.w);
              lo = ice_cell_value_unrimed(cf + 3 * kCellCoefs, a1.w);
            }
            const bool odd = !(dbits(q) < kInfBits && dbits(n) < kInfBits && dbits(m) < kInfBits);
            /* columns 6 and 7: the limits of the number */
            if (fix_below_one(hi, sh.z)) n = d_from_fix(hi, sh.z) * n;
            if (!fix_below_one(lo, sh.w)) n = d_from_fix(lo, sh.w) * n;
            R1[k] = n;
            v1 = d_from_fix(vm, sh.y) * FR[k];
            v2 = d_from_fix(vn, sh.x) * FR[k];
            if (odd) v1 = d_from_bits(kNaNBits);
          }
          if (!dpos(qs)) v1 = d_from_bits(kNaNBits); /* no cloud fraction: reported below */
          lmax = dmax_nn(lmax, v1 * CF[k]);
        }
        V1[k] = v1;
        V2[k] = v2;
      }
      if (k_qxbot < kbot && lane == (k_qxbot + 1 - k_qxtop) % LANES) {
        V1[k_qxbot + 1] = 0; /* the cell receiving the leading edge has no fall speed */
        V2[k_qxbot + 1] = 0;
      }
      const double Co_max = group_max_wide<LANES, SPLIT>(mask, gs, lmax) * dt_left;
      if (!(Co_max >= 0) || Co_max > 2.0e9) {
        err |= kErrNumeric;
        break;
      }

      /* generalized_sedimentation + calc_first_order_upwind_step (kdir = -1):
       * fluxes from start-of-substep values, inflow from the level above by a
       * shuffle (carried across chunks), zero inflow at k_qxtop. */
      const int tmpint1 = static_cast<int>(Co_max + 1);
      const double dt_sub = ddiv_int(dt_left, double(tmpint1));
      const int k_temp = (k_qxbot == kbot) ? k_qxbot : k_qxbot + 1;
      double carry0 = 0, carry1 = 0, carry2 = 0, carry3 = 0, flux_bot = 0;
      for (int base = k_qxtop; base <= k_temp; base += LANES) {
        const int k = base + lane;
        const bool act = k <= k_temp;
        double r0 = 0, r1 = 0, r2 = 0, r3 = 0, f0 = 0, f1 = 0, f2 = 0, f3 = 0;
        if (act) {
          const double v1 = V1[k];
          r0 = R0[k];
          r1 = R1[k];
          f0 = v1 * r0;
          if (number) f1 = V2[k] * r1;
          if (sp == 2) {
            r2 = R2[k];
            r3 = R3[k];
            f2 = v1 * r2;
            f3 = v1 * r3;
          }
        }
        /* no rime in the chunk and none from above: its two fields stay 0 */
        const bool rime = sp == 2 && (LANES > 32 || __any_sync(mask, dnz(r2) || dnz(r3) || dnz(carry2) || dnz(carry3)));
        double u0 = __shfl_up_sync(mask, f0, 1, kWarp), u1 = 0, u2 = 0, u3 = 0;
        if (number) u1 = __shfl_up_sync(mask, f1, 1, kWarp);
        if (rime) {
          u2 = __shfl_up_sync(mask, f2, 1, kWarp);
          u3 = __shfl_up_sync(mask, f3, 1, kWarp);
        }
        if constexpr (LANES > 32) {
          double* const edge = gs->edge[group_warp<LANES>()];
          if ((lane & 31) == 31) {
            edge[0] = f0; edge[1] = f1; edge[2] = f2; edge[3] = f3;
          }
          group_sync<LANES, SPLIT>(mask);
          if ((lane & 31) == 0 && lane > 0) {
            u0 = edge[-4]; u1 = edge[-3]; u2 = edge[-2]; u3 = edge[-1];
          }
        }
        if (lane == 0) {
          u0 = carry0; u1 = carry1; u2 = carry2; u3 = carry3;
        }
        if (act) {
          const double c = CF[k] * dt_sub;
          R0[k] = fma(u0 - f0, c, r0);
          if (number) R1[k] = fma(u1 - f1, c, r1);
          if (rime) {
            R2[k] = fma(u2 - f2, c, r2);
            R3[k] = fma(u3 - f3, c, r3);
          }
          if (sp == 1) PF[k + 1] += f0;
          if (k == kbot) flux_bot = f0;
        }
        if (base + LANES <= k_temp) {
          carry0 = __shfl_sync(mask, f0, kWarp - 1, kWarp);
          if (number) carry1 = __shfl_sync(mask, f1, kWarp - 1, kWarp);
          if (rime) {
            carry2 = __shfl_sync(mask, f2, kWarp - 1, kWarp);
            carry3 = __shfl_sync(mask, f3, kWarp - 1, kWarp);
          }
        }
      }
      if (k_qxbot == kbot) {
        /* a group of several warps: the lane that owns the bottom level sums */
        if constexpr (LANES <= 32) flux_bot = __shfl_sync(mask, flux_bot, (kbot - k_qxtop) % LANES, LANES);
        prt_accum += flux_bot * dt_sub;
      } else {
        k_qxbot += 1;
      }
      dt_left -= dt_sub;
      first = false;
    }
    if constexpr (LANES > 32) {
      if (lane == kbot - k_qxtop) gs->prt[sp] = prt_accum;
      group_sync<LANES, SPLIT>(mask);
      prt_accum = gs->prt[sp];
    }
    if (sp == 0) precip_liq_surf = prt_accum * C::INV_RHO_H2O * inv_dt;
    else if (sp == 1) precip_liq_surf += prt_accum * C::INV_RHO_H2O * inv_dt;
    else precip_ice_surf += prt_accum * C::INV_RHO_H2O * inv_dt;

    group_sync<LANES, SPLIT>(mask);
    for (int k = k_qxtop + lane; k <= k_qxbot; k += LANES) {
      g0[co + k] = R0[k];
      g1[co + k] = R1[k];
      if (sp == 2) {
        in.qm[co + k] = R2[k];
        in.bm[co + k] = R3[k];
      }
    }
    if (sp == 1) {
      /* interfaces above the top stay at part1's zero */
      for (int k = k_qxtop + 1 + lane; k <= nk; k += LANES) in.precip_liq_flux[ci + k] = PF[k];
    }
    group_sync<LANES, SPLIT>(mask);
  };
  if constexpr (SPLIT) {
    const int sp = int(threadIdx.x) / LANES;
    if (sp == 0) species(std::integral_constant<int, 0>{});
    else if (sp == 1) species(std::integral_constant<int, 1>{});
    else species(std::integral_constant<int, 2>{});
    __syncthreads();
    if (threadIdx.x == 0) {
      /* thread 0 belongs to the first group: gs[0], gs[1], gs[2] are the three */
      precip_liq_surf = gs[0].prt[0] * C::INV_RHO_H2O * inv_dt;
      precip_liq_surf += gs[1].prt[1] * C::INV_RHO_H2O * inv_dt;
      precip_ice_surf = gs[2].prt[2] * C::INV_RHO_H2O * inv_dt;
    }
  } else {
    species(std::integral_constant<int, 0>{});
    species(std::integral_constant<int, 1>{});
    species(std::integral_constant<int, 2>{});
  }
  if (SPLIT ? threadIdx.x == 0 : lane == 0) {
    in.precip_liq_surf[col] = precip_liq_surf;
    in.precip_ice_surf[col] = precip_ice_surf;
  }
}

/* K2 of the FP32-bulk form.  Same algorithm and order as p3_sed.  Fall
 * speeds, density, fall-speed factors, 1/dz and an FP32 shadow of each
 * species field live in FP32 shared arrays and drive the fluxes; the Courant
 * maximum is taken in FP32.
 *
 * The accumulation of the flux divergence is carried by time-integrated face
 * fluxes: G_k = sum over substeps of F_k dt_sub, the flux leaving level k
 * downward, kept as a double-float (~48 significant bits).  A level's FP64
 * state after any number of substeps is R_k = B_k + (g / dpres_k) (G_{k-1} -
 * G_k), with B_k its value at the start (kept in the species' global array).
 * So a substep costs one double-float multiply-add (FP32 instructions only)
 * per field and level; both neighbours of a face read the same G, so the
 * column's mass telescopes exactly, and the surface precipitation is the
 * bottom face's G.  Where a limiter rewrites a level's state to x during the
 * walk, B_k is reset so that R_k = x at that moment.
 *
 * What bounds it: latency, at 20 warps an SM (issue 54 %, FP64 pipe 42 %).  The
 * compiler keeps global reads behind the stores in front of them, which may
 * alias, so each would wait for memory by itself; they are therefore grouped by
 * hand: the density a chunk ahead in the flux walk, two chunks at a time where a
 * species is read, all fields of a chunk at once where its state is rebuilt.
 * 345,600 x 128 9.30 -> 8.05 ms, 21,600 x 128 822 -> 727 us. */
template <int LANES, bool SPLIT = false>
__device__ void p3_sed_bulk(const Inst& in, const int col, const KParams<float>& kp, const Tabs<float>& tb,
                            double* __restrict__ sm, GroupScratch* gs, uint32_t& err) {
  if (in.cflag[col] == 0) return;
  const RuntimeDev& rt = kp.rt;
  const unsigned mask = 0xffffffffu;
  const int lane = threadIdx.x & (LANES - 1);
  const int nk = in.nlev;
  const int S = kp.sm_stride;
  const int64_t co = int64_t(col) * in.ld;
  const int64_t ci = int64_t(col) * in.ld_int;
  const double dt = in.dt;
  const double inv_dt = 1 / dt;
  const bool predictNc = in.predictNc != 0;
  const int kbot = nk - 1;
  constexpr int kWarp = 32; /* lanes that shuffle with one another */
#define SMA(a, k) sm[(a)*S + (k)]
  /* kSedBulkSlots slots of S doubles; two float arrays share a slot.  The
   * density is read from the hand-over row (a float per level, L1-resident
   * during the walk) rather than held in a slot. */
  const float* const RHOf = scr_f(in, S_RHO, col);
  float* const FACf = reinterpret_cast<float*>(&SMA(0, 0));
  float* const CLDf = FACf + S;
  double* const COEF = &SMA(1, 0); /* g / dpres */
  float* const INVDZf = reinterpret_cast<float*>(&SMA(2, 0));
  float* const COEFf = INVDZf + S;
  /* Fields in pairs for the packed FP32 instructions: FP32 shadows of
   * fields (0, 1) and (2, 3), the fall speeds (V1, V2), and the time-
   * integrated face fluxes of fields (0, 1) and (2, 3) as double-floats
   * {hi_a, hi_b, lo_a, lo_b} (two slots each). */
  float2* const R23 = reinterpret_cast<float2*>(&SMA(3, 0));
  float2* const V12 = reinterpret_cast<float2*>(&SMA(4, 0));
  float2* const R01 = reinterpret_cast<float2*>(&SMA(5, 0));
  float4* const G01 = reinterpret_cast<float4*>(&SMA(6, 0));
  float4* const G23 = reinterpret_cast<float4*>(&SMA(8, 0));
  float2* const PF = reinterpret_cast<float2*>(G23); /* rain flux sum (rain has two fields) */
  /* the double-float G of field f at level k, as a double */
  auto g_value = [&](int f, int k) -> double {
    const float4 g = (f < 2 ? G01 : G23)[k];
    return (f & 1) ? dfloat_value(make_float2(g.y, g.w)) : dfloat_value(make_float2(g.x, g.z));
  };
  auto r_set = [&](int f, int k, float v) {
    float2& r = (f < 2 ? R01 : R23)[k];
    if (f & 1) {
      r.y = v;
    } else {
      r.x = v;
    }
  };
  /* Top and bottom of the three species (p3_find_impl.hpp) in one pass on
   * the integer pipes.  A species only ever changes the levels from its top
   * down to its final leading edge, so conversions, flux coefficients and the
   * FP64 state rebuild are limited to those levels; the levels above the top
   * and below the leading edge keep their values. */
  int top[3] = {1 << 30, 1 << 30, 1 << 30}, bot[3] = {-1, -1, -1};
  for (int k = lane; k < nk; k += LANES) {
    if (dge(in.qc[co + k], C::QSMALL)) { top[0] = min(top[0], k); bot[0] = k; }
    if (dge(in.qr[co + k], C::QSMALL)) { top[1] = min(top[1], k); bot[1] = k; }
    if (dge(in.qi[co + k], C::QSMALL)) { top[2] = min(top[2], k); bot[2] = k; }
  }
  if (SPLIT && lane < 3) gs->prt[lane] = 0;
  group_bounds<LANES, SPLIT>(mask, gs, top, bot);
  const int k_first = min(top[0], min(top[1], top[2]));
  constexpr int kBatch = LANES > 32 ? 1 : 2; /* chunks read at once */
  for (int k = k_first + lane; k < nk; k += kBatch * LANES) {
    double dp[kBatch], dz[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      dp[i] = in.dpres[co + min(k + i * LANES, kbot)];
      dz[i] = in.dz[co + min(k + i * LANES, kbot)];
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int ki = min(k + i * LANES, kbot);
      const double coef = C::gravit * rcp_newton(dp[i]);
      INVDZf[ki] = 1.0f / float(dz[i]);
      COEF[ki] = coef;
      COEFf[ki] = float(coef);
    }
  }
  double precip_liq_surf = 0, precip_ice_surf = 0;

  /* The three species, each with its code specialised (field count, tables,
   * limiters) at compile time. */
  auto species = [&](auto sp_tag) {
    constexpr int sp = decltype(sp_tag)::value;
    double* const B0 = sp == 0 ? in.qc : (sp == 1 ? in.qr : in.qi);
    double* const B1 = sp == 0 ? in.nc : (sp == 1 ? in.nr : in.ni);
    double* const B2 = in.qm;
    double* const B3 = in.bm;
    double* const Bf[4] = {B0, B1, B2, B3};
    const double* cldp = sp == 0 ? in.cld_frac_l : (sp == 1 ? in.cld_frac_r : in.cld_frac_i);
    const int sfac = sp == 0 ? S_ACN : (sp == 1 ? S_RHOFACR : S_RHOFACI);
    const float* const facp = scr_f(in, sfac, col);
    const int nfield = sp == 0 ? (predictNc ? 2 : 1) : (sp == 1 ? 2 : 4);
    const int nstate = sp == 2 ? 4 : 2; /* fields that limiters may rewrite */
    /* (the species of a split group run at once: the rows are the ice's) */
    constexpr bool kDefer = sp == 2 || (sp == 1 && !SPLIT);
    float* const late_vn = scr_f(in, S_RHO, col) + in.ld;
    float* const late_gh = scr_f(in, S_RHOFACR, col) + in.ld;
    float* const late_gl = scr_f(in, S_RHOFACI, col) + in.ld;
    float* const late_vb = scr_f(in, S_ACN, col) + in.ld;
    const float kNotLate = __uint_as_float(0xffc0deadu);
    /* R_k := x = v cldf now (k owned by this lane; G_{k-1} belongs to the lane
     * above and is final for this substep after the warp barrier): the shadow
     * becomes x rounded and B_k = x - (g / dpres_k) (G_{k-1} - G_k). */
    auto reset_value = [&](int k, float v, float cldf, double gin, double g) {
      return fma(-COEF[k], gin - g, f2d(v) * f2d(cldf));
    };
    auto set_state = [&](int f, int k, float v, float cldf) {
      const double gin = k > 0 ? g_value(f, k - 1) : 0.0;
      Bf[f][co + k] = reset_value(k, v, cldf, gin, g_value(f, k));
      r_set(f, k, __fmul_rn(v, cldf));
    };
    /* The number and the rime volume are reset every other substep somewhere
     * in a chunk (30 times per column in all, a dozen FP64 instructions each,
     * for a few lanes), and only the last reset of a level counts.  So a reset
     * of these fields records v and both G, and the rebuild forms B_k once:
     * G_k in the dead B_k's place, v and the number's G_{k-1} in the unused
     * halves of the hand-over rows, the volume's G_{k-1} in rho_qi (which part1
     * left at 0 and part3 writes).  The same roundings, so the same state;
     * 1.03 -> 0.94 ms at 21,600 x 128, 85 -> 70 us at 64 x 72. */
    auto defer_state = [&](int f, int k, float v, float cldf) {
      const float4 g = (f < 2 ? G01 : G23)[k];
      const float4 gin = k > 0 ? (f < 2 ? G01 : G23)[k - 1] : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float2*>(&Bf[f][co + k]) = make_float2(g.y, g.w);
      if (f == 1) {
        late_vn[k] = v;
        late_gh[k] = gin.y;
        late_gl[k] = gin.w;
      } else {
        late_vb[k] = v;
        *reinterpret_cast<float2*>(&in.rho_qi[co + k]) = make_float2(gin.y, gin.w);
      }
      r_set(f, k, __fmul_rn(v, cldf));
    };

    const int k_qxtop = top[sp];
    int k_qxbot = bot[sp];
    if (k_qxbot < 0) return; /* species absent (group-uniform) */
    /* the walk and the rebuild read G one level above the top */
    /* kBatch chunks are read before any is stored */
    for (int k = max(k_qxtop - 1, 0) + lane; k < nk; k += kBatch * LANES) {
      double b0[kBatch], b1[kBatch], b2[kBatch], b3[kBatch], cl[kBatch];
      float fac[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int64_t o = co + min(k + i * LANES, kbot);
        b0[i] = B0[o];
        b1[i] = B1[o];
        cl[i] = cldp[o];
        fac[i] = facp[min(k + i * LANES, kbot)];
        if (sp == 2) {
          b2[i] = B2[o];
          b3[i] = B3[o];
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int ki = k + i * LANES;
        if (ki >= nk) break;
        G01[ki] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (sp == 2) G23[ki] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ki < k_qxtop) continue;
        R01[ki] = make_float2(float(b0[i]), float(b1[i]));
        CLDf[ki] = float(cl[i]);
        FACf[ki] = fac[i];
        if (kDefer) late_vn[ki] = kNotLate;
        if (sp == 2) {
          R23[ki] = make_float2(float(b2[i]), float(b3[i]));
          late_vb[ki] = kNotLate;
        }
      }
    }
    if (sp == 1) {
      for (int k = k_qxtop + 1 + lane; k <= nk; k += LANES) PF[k] = make_float2(0.f, 0.f);
    }
    group_sync<LANES, SPLIT>(mask);

    /* The substep schedule is FP32 scalar work: one dt_sub scales every face
     * flux of a substep alike, so its rounding only changes that substep's
     * length by ~1e-7 relative and leaves the mass budget exact. */
    float dt_left = float(dt);
    bool first = true;
    int nsub = 0;
    while (dt_left > float(C::dt_left_tol)) {
      if (++nsub > kMaxSubsteps) {
        err |= kErrSubstep;
        break;
      }
      float lmax = 0.0f; /* max of V / dz; the Courant number is that times dt_left */
      for (int k = k_qxtop + lane; k <= k_qxbot; k += LANES) {
        float v1 = 0, v2 = 0;
        bool fall = false;
        /* In-cloud values in FP32.  The first substep applies the reference's
         * thresholds and limits (and the bm quirk: bm_incld uses 1/cld_frac_l);
         * the FP64 state is rewritten wherever a limiter made an in-cloud value
         * differ from the plain one. */
        const float cldf = CLDf[k];
        const float icf = 1.0f / cldf;
        if (sp == 0) {
          const float2 r01 = R01[k];
          const float n_plain = r01.y * icf;
          float qc_f = r01.x * icf, n_in = n_plain;
          if (first) {
            if (dge(B0[co + k], C::QSMALL)) {
              n_in = vmax(n_in, 0.0f);
            } else {
              qc_f = 0;
              n_in = 0;
            }
            qc_f = vmin(qc_f, float(C::incloud_limit));
          }
          if (qc_f > float(C::QSMALL)) {
            float mu_c, lamc;
            float n_out = n_in;
            get_cloud_dsd2<float>(qc_f, n_out, mu_c, RHOf[k], lamc);
            if (n_out != n_plain) set_state(1, k, n_out, cldf);
            const float dum = 1.0f / (lamc * lamc);
            v1 = FACf[k] * ((5.0f + mu_c) * (4.0f + mu_c)) * dum;
            if (predictNc) v2 = FACf[k] * ((2.0f + mu_c) * (1.0f + mu_c)) * dum;
            fall = true;
          }
        } else if (sp == 1) {
          const float2 r01 = R01[k];
          const float n_plain = r01.y * icf;
          float qr_f = r01.x * icf, n_in = n_plain;
          if (first) {
            if (dge(B0[co + k], C::QSMALL)) {
              n_in = vmax(n_in, 0.0f);
            } else {
              qr_f = 0;
              n_in = 0;
            }
            qr_f = vmin(qr_f, float(C::precip_limit));
          }
          if (qr_f > float(C::QSMALL)) {
            float mu_r = 0, lamr;
            float n_out = n_in;
            get_rain_dsd2<float>(qr_f, n_out, mu_r, lamr, rt);
            Table3<float> t3;
            lookup3<float>(mu_r, lamr, rt, t3);
            v1 = apply_table3<float>(tb, tb.vm, t3) * FACf[k];
            v2 = apply_table3<float>(tb, tb.vn, t3) * FACf[k];
            if (n_out != n_plain) {
              if constexpr (kDefer) {
                defer_state(1, k, n_out, cldf);
              } else {
                set_state(1, k, n_out, cldf);
              }
            }
            fall = true;
          }
        } else {
          const float2 r01 = R01[k], r23 = R23[k];
          const float ni_plain = r01.y * icf, qm_plain = r23.x * icf, bm_plain = r23.y * icf;
          float qi_f = r01.x * icf, ni_f = ni_plain, qm_f = qm_plain, bm_f = bm_plain;
          if (first) {
            if (dge(B0[co + k], C::QSMALL)) {
              ni_f = vmax(ni_f, 0.0f);
            } else {
              qi_f = 0;
              ni_f = 0;
            }
            if (dge(B0[co + k], C::QSMALL) && dge(B2[co + k], C::QSMALL)) {
              bm_f = vmax(r23.y * (1.0f / float(in.cld_frac_l[co + k])), 0.0f);
            } else {
              qm_f = 0;
              bm_f = 0;
            }
            qi_f = vmin(qi_f, float(C::incloud_limit));
            bm_f = vmin(bm_f, float(C::incloud_limit));
          }
          const bool present = qi_f > float(C::QSMALL);
          /* ice without rime in the whole chunk: no rime density, and two table
           * corners instead of eight (with the fluxes below 345,600 x 128 10.04 ->
           * 9.29 ms, 21,600 x 128 900 -> 822 us; a bit per chunk kept from substep
           * to substep instead of the votes: 9.55 ms; the vote over all lanes ahead
           * of the loop body 4 % slower) */
          const bool rime = LANES > kWarp || __any_sync(chunk_mask(k - lane, k_qxbot),
                                                        present && (r23.x != 0.f || r23.y != 0.f));
          if (present) {
            const float ni_l = vmax(ni_f, float(C::NSMALL));
            float tv[4]; /* columns 0, 1, 6, 7, packed copy */
            if (rime) {
              const float rhop = calc_bulk_rho_rime<float>(qi_f, qm_f, bm_f, rt);
              if (qm_f != qm_plain) set_state(2, k, qm_f, cldf);
              if (bm_f != bm_plain) defer_state(3, k, bm_f, cldf);
              TableIce<float> ti;
              lookup_ice<float>(qi_f, ni_l, qm_f, rhop, ti);
              ice_table4_f32<kIceSedCols>(tb.ice, ti, 0, tv);
            } else {
              ice_table4_unrimed<kIceSedCols>(tb.ice, qi_f, ni_l, 0, tv);
            }
            float n2 = vmin(ni_l, tv[2] * ni_l);
            n2 = vmax(n2, tv[3] * n2);
            if (n2 != ni_plain) defer_state(1, k, n2, cldf);
            const float f = rt.f.ice_sedimentation_factor * FACf[k];
            v1 = f * tv[1];
            v2 = f * tv[0];
            fall = true;
          }
        }
        V12[k] = make_float2(v1, v2);
        if (fall) lmax = vmax(lmax, v1 * INVDZf[k]);
      }
      if (k_qxbot < kbot && lane == (k_qxbot + 1 - k_qxtop) % LANES) {
        V12[k_qxbot + 1] = make_float2(0.f, 0.f); /* the cell receiving the leading edge has no fall speed */
      }
      /* the density row has no slot and little L1 beside the shared memory: read a
       * chunk ahead of its use */
      float rho_next = RHOf[min(k_qxtop + lane, kbot)];
      const float Co_max = group_max_wide<LANES, SPLIT>(mask, gs, lmax) * dt_left;
      if (!(Co_max >= 0.0f) || Co_max > 2.0e9f) {
        err |= kErrNumeric;
        break;
      }
      const int tmpint1 = static_cast<int>(Co_max + 1.0f);
      const float dt_sub = dt_left / float(tmpint1);
      const int k_temp = (k_qxbot == kbot) ? k_qxbot : k_qxbot + 1;
      /* FP32 fluxes from the shadows; double-float time-integrated face
       * fluxes; the shadows follow with the FP32 flux divergence.  Fields go
       * in pairs through the packed FP32 instructions (same operations and
       * rounding as the scalar form). */
      float2 c01 = make_float2(0.f, 0.f), c23 = make_float2(0.f, 0.f);
      for (int base = k_qxtop; base <= k_temp; base += LANES) {
        const int k = base + lane;
        const bool act = k <= k_temp;
        float2 f01 = make_float2(0.f, 0.f), f23 = make_float2(0.f, 0.f);
        const float rho = rho_next;
        if (base + LANES <= k_temp) rho_next = RHOf[min(k + LANES, kbot)];
        if (act) {
          const float2 rho2 = f2splat(rho);
          const float2 v = V12[k];
          f01 = __fmul2_rn(__fmul2_rn(v, R01[k]), rho2);
          if (nfield < 2) f01.y = 0.f;
          if (nfield > 2) f23 = __fmul2_rn(__fmul2_rn(f2splat(v.x), R23[k]), rho2);
        }
        /* no rime falls in the chunk or comes from above: its fields stay as they are */
        const bool rime = nfield > 2 && (LANES > 32 || __any_sync(mask, f23.x != 0.f || f23.y != 0.f || c23.x != 0.f ||
                                                                           c23.y != 0.f));
        float2 u01, u23 = make_float2(0.f, 0.f);
        u01.x = __shfl_up_sync(mask, f01.x, 1, kWarp);
        u01.y = nfield > 1 ? __shfl_up_sync(mask, f01.y, 1, kWarp) : 0.f;
        if (rime) {
          u23.x = __shfl_up_sync(mask, f23.x, 1, kWarp);
          u23.y = __shfl_up_sync(mask, f23.y, 1, kWarp);
        }
        if constexpr (LANES > 32) {
          float4* const edge = reinterpret_cast<float4*>(gs->edge[group_warp<LANES>()]);
          if ((lane & 31) == 31) *edge = make_float4(f01.x, f01.y, f23.x, f23.y);
          group_sync<LANES, SPLIT>(mask);
          if ((lane & 31) == 0 && lane > 0) {
            const float4 u = *reinterpret_cast<const float4*>(gs->edge[group_warp<LANES>() - 1]);
            u01 = make_float2(u.x, u.y);
            u23 = make_float2(u.z, u.w);
          }
        }
        if (lane == 0) {
          u01 = c01;
          u23 = c23;
        }
        if (act) {
          const float2 coef2 = f2splat(COEFf[k] * dt_sub);
          dfloat2_add_prod(G01[k], f01, dt_sub);
          R01[k] = __ffma2_rn(__fadd2_rn(u01, f2neg(f01)), coef2, R01[k]);
          if (rime) {
            dfloat2_add_prod(G23[k], f23, dt_sub);
            R23[k] = __ffma2_rn(__fadd2_rn(u23, f2neg(f23)), coef2, R23[k]);
          }
          if (sp == 1) dfloat_add(PF[k + 1], f01.x);
        }
        if (base + LANES <= k_temp) {
          c01.x = __shfl_sync(mask, f01.x, kWarp - 1, kWarp);
          c01.y = nfield > 1 ? __shfl_sync(mask, f01.y, kWarp - 1, kWarp) : 0.f;
          if (rime) {
            c23.x = __shfl_sync(mask, f23.x, kWarp - 1, kWarp);
            c23.y = __shfl_sync(mask, f23.y, kWarp - 1, kWarp);
          }
        }
      }
      if (k_qxbot < kbot) k_qxbot += 1;
      dt_left -= dt_sub;
      first = false;
      group_sync<LANES, SPLIT>(mask); /* G of the level above is read by set_state */
    }
    group_sync<LANES, SPLIT>(mask);
    /* the bottom face's integral is what left the column: V is zero at the
     * leading edge, so G_kbot gains only in substeps where the species
     * reaches the surface */
    const double prt_accum = g_value(0, kbot);
    if (SPLIT && lane == 0) gs->prt[sp] = prt_accum;
    if (sp == 0) precip_liq_surf = prt_accum * C::INV_RHO_H2O * inv_dt;
    else if (sp == 1) precip_liq_surf += prt_accum * C::INV_RHO_H2O * inv_dt;
    else precip_ice_surf += prt_accum * C::INV_RHO_H2O * inv_dt;

    /* FP64 state: R_k = B_k + (g / dpres_k) (G_{k-1} - G_k), on the levels
     * from the top to the final leading edge (G is zero elsewhere) */
    /* G_{k-1} comes from the lane above (the same value that lane forms for
     * its own level); above the top it is zero: no flux enters there */
    double g_in[4] = {0.0, 0.0, 0.0, 0.0};
    for (int base = k_qxtop; base <= k_qxbot; base += LANES) {
      const int k = base + lane;
      const bool act = k <= k_qxbot;
      const int kc = min(k, kbot);
      /* read at once: a field's store would hold up the next field's reads */
      double B[4];
      float late_n = kNotLate, late_b = kNotLate;
#pragma unroll
      for (int f = 0; f < nstate; ++f) B[f] = read_now(&Bf[f][co + kc]);
      if (kDefer) late_n = read_now(&late_vn[kc]);
      if (sp == 2) late_b = read_now(&late_vb[kc]);
      bool rime = sp == 2;
      if (sp == 2 && LANES == 32) {
        const float4 g = G23[kc];
        rime = __any_sync(mask, act && (g.x != 0.f || g.y != 0.f || __float_as_uint(late_b) != 0xffc0deadu)) ||
               dnz(g_in[2]) || dnz(g_in[3]);
      }
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        if (f < nstate && (f < 2 || rime)) {
          const double g = act ? g_value(f, k) : 0.0;
          double gin = __shfl_up_sync(mask, g, 1, kWarp);
          if (lane == 0) gin = g_in[f];
          if (LANES > 32 && (lane & 31) == 0 && lane > 0 && act) gin = g_value(f, k - 1);
          if (act) {
            const float v = f == 1 ? late_n : late_b;
            if (kDefer && (f == 1 || f == 3) && __float_as_uint(v) != 0xffc0deadu) {
              const float2 g0 = make_float2(__int_as_float(__double2loint(B[f])), __int_as_float(__double2hiint(B[f])));
              float2 gin0;
              if (f == 1) {
                gin0 = make_float2(late_gh[k], late_gl[k]);
              } else {
                gin0 = *reinterpret_cast<const float2*>(&in.rho_qi[co + k]);
                in.rho_qi[co + k] = 0;
              }
              B[f] = reset_value(k, v, CLDf[k], dfloat_value(gin0), dfloat_value(g0));
            }
            Bf[f][co + k] = B[f] + COEF[k] * (gin - g);
          }
          g_in[f] = __shfl_sync(mask, g, kWarp - 1, kWarp);
        }
      }
    }
    if (sp == 1) {
      /* interfaces above the top stay at part1's zero */
      for (int k = k_qxtop + 1 + lane; k <= nk; k += LANES) in.precip_liq_flux[ci + k] = dfloat_value(PF[k]);
    }
    group_sync<LANES, SPLIT>(mask);
  };
  if constexpr (SPLIT) {
    const int sp = int(threadIdx.x) / LANES;
    if (sp == 0) species(std::integral_constant<int, 0>{});
    else if (sp == 1) species(std::integral_constant<int, 1>{});
    else species(std::integral_constant<int, 2>{});
    __syncthreads();
    if (threadIdx.x == 0) {
      /* thread 0 belongs to the first group: gs[0], gs[1], gs[2] are the three */
      precip_liq_surf = gs[0].prt[0] * C::INV_RHO_H2O * inv_dt;
      precip_liq_surf += gs[1].prt[1] * C::INV_RHO_H2O * inv_dt;
      precip_ice_surf = gs[2].prt[2] * C::INV_RHO_H2O * inv_dt;
    }
  } else {
    species(std::integral_constant<int, 0>{});
    species(std::integral_constant<int, 1>{});
    species(std::integral_constant<int, 2>{});
  }
  if (SPLIT ? threadIdx.x == 0 : lane == 0) {
    in.precip_liq_surf[col] = precip_liq_surf;
    in.precip_ice_surf[col] = precip_ice_surf;
  }
#undef SMA
}

/* K3: homogeneous freezing and p3_main_part3 of the levels first + lane, first
 * + step + lane, ... of one column that went on past part2. */
template <class TR, int LANES>
__device__ void p3_part3(const Inst& in, const int col, const KParams<TR>& kp, const Tabs<TR>& tb, const int inst_idx,
                         const int first, const int step, uint32_t& err) {
  if (in.cflag[col] == 0) return;
  const RuntimeDev& rt = kp.rt;
  const int lane = threadIdx.x & (LANES - 1);
  const int nk = in.nlev;
  const int64_t co = int64_t(col) * in.ld;
  const bool do_ice = rt.do_ice_production != 0;
  constexpr bool kF64 = sizeof(TR) == sizeof(double);
  const auto check = [&](const int64_t o, const int k) {
    if (!kp.check) return;
    /* check_values (p3_check_values_impl.hpp:26-81, called at
     * p3_main_impl.hpp:316-323 with T = th exner): T must lie in
     * (173, 323) K and qv in (0, 0.04); the reference traps only on T, and
     * only when its debug abort is on.  Recorded, never trapped. */
    const double qv = in.qv[o], T = in.th[o] * m_div(1.0, in.inv_exner[o]);
    const unsigned long long key = check_key(inst_idx, col, k);
    if (!(dgt(T, 173.0) && dlt(T, 323.0))) {
      atomicAdd(&kp.check[kChkTCount], 1ull);
      atomicMin(&kp.check[kChkTFirst], key);
      if (kp.check_fail) err |= kErrRange;
    }
    if (!(dpos(qv) && dlt(qv, 0.04))) {
      atomicAdd(&kp.check[kChkQvCount], 1ull);
      atomicMin(&kp.check[kChkQvFirst], key);
    }
  };
  /* ---------------- phase 4: homogeneous freezing + p3_main_part3 ---------------- */
  for (int k = first + lane; k < nk; k += step) {
    const int64_t o = co + k;
    /* Everything a level may need is read at once.  The volatile reads keep the
     * compiler from moving them behind the hydrometeor test, which moves fewer
     * bytes but waits for memory twice (FP32-bulk 345,600 x 128 1.85 ms against
     * 1.64; with every output written back on every level 1.82). */
    State s;
    s.qc = in.qc[o]; s.nc = in.nc[o]; s.qr = in.qr[o]; s.nr = in.nr[o];
    s.qi = in.qi[o]; s.qm = in.qm[o]; s.ni = in.ni[o]; s.bm = in.bm[o];
    s.qv = read_now(in.qv + o);
    s.th = read_now(in.th + o);
    const double inv_exner = read_now(in.inv_exner + o);
    const double cld_l = read_now(in.cld_frac_l + o), cld_r = read_now(in.cld_frac_r + o),
                 cld_i = read_now(in.cld_frac_i + o);
    const double t_start = read_now(scr_at(in, S_TATM, col) + k);
    /* rho: FP64 in the plain form, a float in the FP32-bulk hand-over */
    double rho = 0, inv_rho = 0;
    float rho_f = 0.f, inv_rho_f = 0.f;
    if constexpr (kF64) rho = read_now(scr_at(in, S_RHO, col) + k);
    else rho_f = read_now(scr_f(in, S_RHO, col) + k);
    const double vap_in = read_now(in.vap_liq_exchange + o);
    if (!(dge(s.qc, C::QSMALL) || dge(s.qr, C::QSMALL) || dge(s.qi, C::QSMALL))) {
      /* no hydrometeor: what is left goes to vapour, and only what changes is
       * written */
      if (dnz(s.qc) || dnz(s.qr) || dnz(s.qi)) {
        double qv = s.qv, th = s.th, vap_liq = vap_in;
        if (dnz(s.qc)) {
          qv = qv + s.qc;
          th = th - inv_exner * s.qc * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qc;
        }
        if (dnz(s.qr)) {
          qv = qv + s.qr;
          th = th - inv_exner * s.qr * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qr;
        }
        if (dnz(s.qi)) {
          qv = qv + s.qi;
          th = th - inv_exner * s.qi * (C::LatVap + C::LatIce) * C::INV_CP;
        }
        in.qv[o] = qv;
        in.th[o] = th;
        in.vap_liq_exchange[o] = vap_liq;
        in.qc[o] = 0; in.qr[o] = 0; in.qi[o] = 0;
      }
      if (dnz(s.nc)) in.nc[o] = 0;
      if (dnz(s.nr)) in.nr[o] = 0;
      if (dnz(s.ni)) in.ni[o] = 0;
      if (dnz(s.qm)) in.qm[o] = 0;
      if (dnz(s.bm)) in.bm[o] = 0;
      in.rho_qi[o] = 0;
      check(o, k);
      continue;
    }
    if constexpr (kF64) inv_rho = m_div(1.0, rho);
    else inv_rho_f = 1.0f / rho_f;
    double vap_liq = vap_in;
    double eff_qc = 0, eff_qr = 0, eff_qi = 0, rho_qi = 0; /* the first three are stored where formed */
    bool has_c = false, has_r = false, has_i = false;

    /* homogeneous_freezing, p3/impl/p3_ice_sed_impl.hpp:207-270 */
    if (do_ice && dlt(t_start, C::T_homogfrz)) {
      const double Qc_nuc = s.qc, Qr_nuc = s.qr;
      const double Nc_nuc = dmax_c(s.nc, C::NSMALL), Nr_nuc = dmax_c(s.nr, C::NSMALL);
      const bool qc_ge = dge(s.qc, C::QSMALL), qr_ge = dge(s.qr, C::QSMALL);
      if (qc_ge) {
        s.qm = s.qm + Qc_nuc;
        s.qi = s.qi + Qc_nuc;
        s.bm = s.bm + Qc_nuc * C::INV_RHO_RIMEMAX;
        s.ni = s.ni + Nc_nuc;
        s.th = s.th + inv_exner * Qc_nuc * C::LatIce * C::INV_CP;
      }
      if (qr_ge) {
        s.qm = s.qm + Qr_nuc;
        s.qi = s.qi + Qr_nuc;
        s.bm = s.bm + Qr_nuc * C::INV_RHO_RIMEMAX;
        s.ni = s.ni + Nr_nuc;
        s.th = s.th + inv_exner * Qr_nuc * C::LatIce * C::INV_CP;
      }
      if (qc_ge) { s.qc = 0; s.nc = 0; }
      if (qr_ge) { s.qr = 0; s.nr = 0; }
    }

    if constexpr (sizeof(TR) == sizeof(double)) {
      /* part3: cloud */
      if (dge(s.qc, C::QSMALL)) {
        const double qc_incld = m_div(s.qc, cld_l);
        double nc_incld = m_div(s.nc, cld_l);
        TR mu_c, lamc;
        const TR n_in = TR(nc_incld);
        TR n_out = n_in;
        get_cloud_dsd2<TR>(TR(qc_incld), n_out, mu_c, TR(rho), lamc, [](TR x) { return cbrt_fix(x, &kFixTables); });
        apply_n_adjust(nc_incld, n_in, n_out);
        s.nc = nc_incld * cld_l;
        has_c = true;
        eff_qc = double(m_div(TR(0.5) * (mu_c + TR(3)), lamc));
      } else {
        if (dnz(s.qc)) {
          s.qv = s.qv + s.qc;
          s.th = s.th - inv_exner * s.qc * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qc;
        }
        s.qc = 0;
        s.nc = 0;
      }
      /* part3: rain */
      if (dge(s.qr, C::QSMALL)) {
        const double qr_incld = m_div(s.qr, cld_r);
        double nr_incld = m_div(s.nr, cld_r);
        TR mu_r = 0, lamr;
        const TR n_in = TR(nr_incld);
        TR n_out = n_in;
        get_rain_dsd2<TR>(TR(qr_incld), n_out, mu_r, lamr, rt, [](TR x) { return cbrt_fix(x, &kFixTables); });
        apply_n_adjust(nr_incld, n_in, n_out);
        s.nr = nr_incld * cld_r;
        has_r = true;
        eff_qr = double(m_div(TR(1.5), lamr));
      } else {
        if (dnz(s.qr)) {
          s.qv = s.qv + s.qr;
          s.th = s.th - inv_exner * s.qr * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qr;
        }
        s.qr = 0;
        s.nr = 0;
      }
      /* part3: ice */
      {
        const bool qi_gt_small = dge(s.qi, C::QSMALL);
        s.ni = dmax_c(s.ni, C::NSMALL);
        if (qi_gt_small) {
          const double qi_incld = m_div(s.qi, cld_i);
          double ni_incld = m_div(s.ni, cld_i);
          double qm_incld = m_div(s.qm, cld_i);
          double bm_incld = m_div(s.bm, cld_i);
          const double rhop = calc_bulk_rho_rime(qi_incld, qm_incld, bm_incld, rt);
          s.qm = qm_incld * cld_i;
          s.bm = bm_incld * cld_i;
          impose_max_total_ni(ni_incld, rt.max_total_ni, inv_rho);
          /* table position, limits and values in fixed point (part3 0.87 ->
           * 0.37 ms at 21,600 x 128, now 0.28) */
          const IceCell cell = ice_cell(m_div(qi_incld, ni_incld), m_div(qm_incld, qi_incld), rhop, &kFixTables);
          const int64_t* const cf = kp.cell_part3 + size_t(cell.cell) * (kCellCols * kCellCoefs);
          const int4 sh = __ldg(reinterpret_cast<const int4*>(kp.cell_part3_shift) + cell.cell);
          const int64_t hi = ice_cell_value(cf, cell), lo = ice_cell_value(cf + kCellCoefs, cell);
          if (fix_below_one(hi, sh.x)) ni_incld = d_from_fix(hi, sh.x) * ni_incld;
          if (!fix_below_one(lo, sh.y)) ni_incld = d_from_fix(lo, sh.y) * ni_incld;
          has_i = true;
          eff_qi = d_from_fix(ice_cell_value(cf + 2 * kCellCoefs, cell), sh.z);
          rho_qi = d_from_fix(ice_cell_value(cf + 3 * kCellCoefs, cell), sh.w);
          if (cell.odd) ni_incld = eff_qi = rho_qi = d_from_bits(kNaNBits);
          s.ni = ni_incld * cld_i;
          if (dlt(s.qm, C::QSMALL)) {
            s.qm = 0;
            s.bm = 0;
          }
        } else {
          if (dnz(s.qi)) {
            s.qv = s.qv + s.qi;
            s.th = s.th - inv_exner * s.qi * (C::LatVap + C::LatIce) * C::INV_CP;
          }
          s.qi = 0; s.ni = 0; s.qm = 0; s.bm = 0;
        }
      }
    } else {
      /* FP32-bulk part3: in-cloud values, DSDs and the diagnostics in FP32; the
       * FP64 state is rewritten only where a limiter changed an in-cloud value */
      if (dge(s.qc, C::QSMALL)) {
        const float icl = 1.0f / float(cld_l);
        const float qc_f = float(s.qc) * icl;
        const float n_in = float(s.nc) * icl;
        float n_out = n_in, mu_c, lamc;
        get_cloud_dsd2<float>(qc_f, n_out, mu_c, rho_f, lamc);
        if (n_out != n_in) s.nc = f2d_int(n_out) * cld_l;
        has_c = true;
        eff_qc = f2d_int(0.5f * (mu_c + 3.0f) / lamc);
      } else {
        if (dnz(s.qc)) {
          s.qv = s.qv + s.qc;
          s.th = s.th - inv_exner * s.qc * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qc;
        }
        s.qc = 0;
        s.nc = 0;
      }
      if (dge(s.qr, C::QSMALL)) {
        const float icr = 1.0f / float(cld_r);
        const float qr_f = float(s.qr) * icr;
        const float n_in = float(s.nr) * icr;
        float n_out = n_in, mu_r = 0, lamr;
        get_rain_dsd2<float>(qr_f, n_out, mu_r, lamr, rt);
        if (n_out != n_in) s.nr = f2d_int(n_out) * cld_r;
        has_r = true;
        eff_qr = f2d_int(1.5f / lamr);
      } else {
        if (dnz(s.qr)) {
          s.qv = s.qv + s.qr;
          s.th = s.th - inv_exner * s.qr * C::LatVap * C::INV_CP;
          vap_liq = vap_liq - s.qr;
        }
        s.qr = 0;
        s.nr = 0;
      }
      {
        const bool qi_gt_small = dge(s.qi, C::QSMALL);
        s.ni = dmax_c(s.ni, C::NSMALL);
        if (qi_gt_small) {
          const float ici = 1.0f / float(cld_i);
          const float qi_f = float(s.qi) * ici;
          const float ni0 = float(s.ni) * ici;
          const float qm0 = float(s.qm) * ici, bm0 = float(s.bm) * ici;
          float qm_f = qm0, bm_f = bm0;
          const float rhop = calc_bulk_rho_rime<float>(qi_f, qm_f, bm_f, rt);
          if (qm_f != qm0) s.qm = f2d_int(qm_f) * cld_i;
          if (bm_f != bm0) s.bm = f2d_int(bm_f) * cld_i;
          float ni_f = ni0;
          impose_max_total_ni(ni_f, rt.f.max_total_ni, inv_rho_f);
          TableIce<float> ti;
          lookup_ice<float>(qi_f, ni_f, qm_f, rhop, ti);
          float ta[4], te[4];
          apply_table_ice4<float>(tb, ti, 0, ta); /* columns 0, 1, 6, 7 */
          apply_table_ice4<float>(tb, ti, 8, te); /* columns 5, 11, 8, 10 */
          ni_f = vmin(ni_f, ta[2] * ni_f);
          ni_f = vmax(ni_f, ta[3] * ni_f);
          has_i = true;
          eff_qi = f2d_int(te[0]);
          rho_qi = f2d_int(te[1]);
          if (ni_f != ni0) s.ni = f2d_int(ni_f) * cld_i;
          if (dlt(s.qm, C::QSMALL)) {
            s.qm = 0;
            s.bm = 0;
          }
        } else {
          if (dnz(s.qi)) {
            s.qv = s.qv + s.qi;
            s.th = s.th - inv_exner * s.qi * (C::LatVap + C::LatIce) * C::INV_CP;
          }
          s.qi = 0; s.ni = 0; s.qm = 0; s.bm = 0;
        }
      }
    }
    if (dlt(s.qr, C::QSMALL)) s.nr = 0;

    store_state(in, o, s);
    in.vap_liq_exchange[o] = vap_liq;
    if (has_c) in.diag_eff_radius_qc[o] = eff_qc;
    if (has_r) in.diag_eff_radius_qr[o] = eff_qr;
    if (has_i) in.diag_eff_radius_qi[o] = eff_qi;
    in.rho_qi[o] = rho_qi;
    check(o, k);
  }
}

/* ------------------------------------------------------------------ */
/* kernels                                                             */
/* ------------------------------------------------------------------ */

/* Table pointers of a CTA: staged into shared memory (K1, when kp.staged)
 * or the global copies.  Returns the first byte after the staged tables, or
 * nullptr when the staging wait gave up. */
template <class TR>
__device__ __forceinline__ unsigned char* setup_tables(const KParams<TR>& kp, bool stage, unsigned char* smem_raw,
                                                       Tabs<TR>& tb, uint32_t& err) {
  tb.collect = kp.collect;
  if (stage) {
    TR* s_ice = reinterpret_cast<TR*>(smem_raw);
    TR* s_t3 = s_ice + kIceTableElems;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + table_smem_bytes<TR>() - 16);
    if (!stage_tables<TR>(kp, s_ice, s_t3, mbar, err)) return nullptr;
    tb.ice = s_ice;
    tb.vn = s_t3;
    tb.vm = s_t3 + 600;
    tb.revap = s_t3 + 1200;
    tb.t3_stride = 2;
    tb.t3_j0 = kp.rt.t3_dumjj - 1;
    return smem_raw + table_smem_bytes<TR>();
  }
  tb.ice = kp.ice;
  tb.vn = kp.vn;
  tb.vm = kp.vm;
  tb.revap = kp.revap;
  tb.t3_stride = kVT1;
  tb.t3_j0 = 0;
  return smem_raw;
}

/* Runs f(w) for the work items of this warp.  With a counter, a warp takes the
 * next item whenever it has finished its last one, so a warp that drew cheap
 * columns takes more of them and no SM idles behind the slowest column list (a
 * static stride gives every warp a fixed share, and an even stride gives it
 * columns of one parity only).  Without one, warps stride the list. */
template <class F>
__device__ __forceinline__ void for_each_work(uint32_t* ctr, int nwork, int groups_per_block, F&& f) {
  if (ctr) {
    for (;;) {
      uint32_t w = 0;
      if ((threadIdx.x & 31) == 0) w = atomicAdd(ctr, 1u);
      w = __shfl_sync(0xffffffffu, w, 0);
      if (w >= uint32_t(nwork)) break;
      f(int(w));
    }
  } else {
    const int groups_total = gridDim.x * groups_per_block;
    for (int w = blockIdx.x * groups_per_block + int(threadIdx.x >> 5); w < nwork; w += groups_total) f(w);
  }
}

/* Column of work item w (single instance or batched work list). */
template <class TR>
__device__ __forceinline__ const Inst& work_inst(const Inst& inst0, const KParams<TR>& kp, int w, int& col) {
  if (kp.work) {
    const WorkItem wi = kp.work[w];
    col = wi.col;
    return kp.insts[wi.inst];
  }
  col = w;
  return inst0;
}

/* Number of work items from w0 on, below w1, that are neighbouring columns of one
 * instance in order: the warp reads the pool's items at once. */
static_assert(kPoolMaxCols < 32, "a pool's items in one ballot");
__device__ __forceinline__ int work_run(const WorkItem* work, int w0, int w1) {
  const int lane = int(threadIdx.x & 31);
  const WorkItem first = work[w0];
  bool follows = false;
  if (lane < w1 - w0) {
    const WorkItem wi = work[w0 + lane];
    follows = wi.inst == first.inst && wi.col == first.col + lane;
  }
  return __ffs(int(~__ballot_sync(0xffffffffu, follows))) - 1;
}

/* BATCH: a work list of several instances, whose field pointers are read from
 * memory where they are used.  A single instance's are kernel arguments:
 * 345,600 x 128 FP32-bulk 5.13 -> 4.94 ms, 21,600 x 128 FP64 2.35 -> 2.33 (K2 and
 * K3 were not faster so).
 * The FP32-bulk instantiation is held to 128 registers (two CTAs of 256
 * threads per SM; a few dozen bytes spill), which measured 25 % faster than 176
 * registers at one CTA per SM. */
template <class TR, bool BATCH>
__global__ void __launch_bounds__(256, sizeof(TR) == sizeof(float) ? 2 : 1)
    p3_part12_kernel(const Inst inst0, const KParams<TR> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<TR> tb;
  unsigned char* base = setup_tables<TR>(kp, kp.staged != 0, smem_raw, tb, err);
  if (!base) {
    if (threadIdx.x == 0) atomicOr(kp.err, err);
    return;
  }
  uint16_t* const list =
      reinterpret_cast<uint16_t*>(base) + size_t(threadIdx.x >> 5) * pool_list_entries(kp.pool_cols, kp.nlev_max);
  for_each_work(kp.wctr ? kp.wctr + 0 : nullptr, kp.npools, kp.groups_per_block, [&](int i) {
    int w0, w1;
    pool_range(kp, i, w0, w1);
    if constexpr (BATCH) {
      while (w0 < w1) { /* a pool's run of columns of one instance */
        int col;
        const Inst& in = work_inst(inst0, kp, w0, col);
        const int n = work_run(kp.work, w0, w1);
        p3_part12<TR, false>(in, col, n, kp, tb, list, nullptr, err);
        w0 += n;
      }
    } else {
      p3_part12<TR, false>(inst0, w0, w1 - w0, kp, tb, list, nullptr, err);
    }
  });
  if (err) atomicOr(kp.err, err);
}

/* K1 with a CTA per column, where a call has fewer columns than the GPU has
 * room for such CTAs: its time is then the latency of one column.  It takes no
 * work from the counters and zeroes them for K2 and K3, which saves a small call
 * the memory fill in front (2 of 65 us at 64 x 72 FP32-bulk). */
template <class TR>
__global__ void __launch_bounds__(kPart12WideThreads, sizeof(TR) == sizeof(float) ? 4 : 2)
    p3_part12_wide_kernel(const Inst inst0, const KParams<TR> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ PoolScratch ps;
  uint32_t err = 0;
  Tabs<TR> tb;
  setup_tables<TR>(kp, false, smem_raw, tb, err);
  if (kp.wctr && blockIdx.x == 0 && threadIdx.x < kWorkCounters) kp.wctr[threadIdx.x] = 0;
  for (int w = blockIdx.x; w < kp.nwork; w += gridDim.x) {
    int col;
    const Inst& in = work_inst(inst0, kp, w, col);
    p3_part12<TR, true>(in, col, 1, kp, tb, reinterpret_cast<uint16_t*>(smem_raw), &ps, err);
  }
  if (err) atomicOr(kp.err, err);
}

/* 96 registers (a few dozen bytes spill): five 4-column CTAs per SM instead of
 * four, 3.61 -> 3.48 ms at 21,600 x 128 (80 registers: no faster). */
template <class TR, int LANES>
__global__ void __maxnreg__(96) p3_sed_kernel(const Inst inst0, const KParams<TR> kp) {
  static_assert(sizeof(TR) == sizeof(double), "the FP32-bulk sedimentation kernel is p3_sed_bulk_kernel");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<TR> tb;
  setup_tables<TR>(kp, false, smem_raw, tb, err);
  const int g_in_block = threadIdx.x / LANES;
  double* sm = reinterpret_cast<double*>(smem_raw) + size_t(g_in_block) * sed_slots<TR>() * kp.sm_stride;
  for_each_work(kp.wctr ? kp.wctr + 1 : nullptr, kp.nwork, kp.groups_per_block, [&](int w) {
    int col;
    const Inst& in = work_inst(inst0, kp, w, col);
    p3_sed<TR, LANES>(in, col, kp, tb, sm, nullptr, err);
  });
  if (err) atomicOr(kp.err, err);
}

/* K2 with a CTA per column, for calls whose columns leave most warps idle
 * (sed_wide_lanes): every level has its own thread of LANES, so a substep costs
 * one fall-speed pass and one flux pass instead of one of each per 32 levels,
 * and with SPLIT the three species, which are independent, run at once.  The
 * calls it is for are bound by the latency of the slowest column's substeps:
 * 64 x 72 FP64 152 -> 109 us, with SPLIT 70 us; FP32-bulk 70 -> 50 -> 33 us. */
template <int LANES, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 3 * LANES : LANES)
    p3_sed_wide_kernel(const Inst inst0, const KParams<double> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<double> tb;
  setup_tables<double>(kp, false, smem_raw, tb, err);
  constexpr int kGroups = SPLIT ? 3 : 1;
  const int g = SPLIT ? int(threadIdx.x) / LANES : 0;
  GroupScratch* const gs = reinterpret_cast<GroupScratch*>(smem_raw);
  double* const sm = reinterpret_cast<double*>(smem_raw + kGroups * sizeof(GroupScratch)) +
                     size_t(g) * sed_slots<double>() * kp.sm_stride;
  int col;
  const Inst& in = work_inst(inst0, kp, int(blockIdx.x), col);
  p3_sed<double, LANES, SPLIT>(in, col, kp, tb, sm, gs + g, err);
  if (err) atomicOr(kp.err, err);
}

/* Tables of the FP32-bulk sedimentation: compact copies, so that the lookups
 * of the substep walk stay in the L1 data cache beside the CTAs' shared memory:
 * the four ice-table columns of sedimentation (16 KB) and the two-column
 * Table3 slices of the rain shape (2.4 KB each) rather than the full tables
 * (48 KB and 12 KB). */
__device__ __forceinline__ void sed_tables(const KParams<float>& kp, Tabs<float>& tb) {
  tb.collect = kp.collect;
  tb.ice = kp.ice_sed;
  tb.vn = kp.t3slice;
  tb.vm = kp.t3slice + kT3SliceElems / 3;
  tb.revap = kp.t3slice + 2 * (kT3SliceElems / 3);
  tb.t3_stride = 2;
  tb.t3_j0 = kp.rt.t3_dumjj - 1;
}

/* K2 of the FP32-bulk form.  STAGED: one CTA of up to 20 columns per SM with
 * the ice table's four columns and the rain slices copied to shared memory
 * first (20.8 KB), for launches that fill every SM; otherwise 4-column CTAs that
 * read them through L1, where a quarter of the gathers missed (the walk waits
 * on them): 0.946 -> 0.899 ms at 21,600 x 128, 10.6 -> 10.1 ms at 345,600 x 128.
 * Held to 96 registers: with its 10 shared slots
 * per column that is five 4-column CTAs (20 warps) per SM, where the
 * latency-bound substep walk gains from every resident warp.  At most 640
 * threads per CTA (the launch checks it). */
template <int LANES, bool STAGED>
__global__ void __maxnreg__(96) p3_sed_bulk_kernel(const Inst inst0, const KParams<float> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<float> tb;
  sed_tables(kp, tb);
  unsigned char* columns = smem_raw;
  if constexpr (STAGED) {
    /* ice table, then vn and vm (sed_table_bytes) */
    float4* const st = reinterpret_cast<float4*>(smem_raw);
    const float4* const ice = reinterpret_cast<const float4*>(tb.ice);
    const float4* const rain = reinterpret_cast<const float4*>(tb.vn);
    constexpr int n_ice = kSedIceElems / 4, n_rain = 2 * (kT3SliceElems / 3) / 4;
    for (int i = threadIdx.x; i < n_ice; i += blockDim.x) st[i] = __ldg(ice + i);
    for (int i = threadIdx.x; i < n_rain; i += blockDim.x) st[n_ice + i] = __ldg(rain + i);
    __syncthreads();
    tb.ice = reinterpret_cast<const float*>(st);
    tb.vn = tb.ice + kSedIceElems;
    tb.vm = tb.vn + kT3SliceElems / 3;
    columns += sed_table_bytes();
  }
  const int g_in_block = threadIdx.x / LANES;
  double* sm = reinterpret_cast<double*>(columns) + size_t(g_in_block) * kSedBulkSlots * kp.sm_stride;
  for_each_work(kp.wctr ? kp.wctr + 1 : nullptr, kp.nwork, kp.groups_per_block, [&](int w) {
    int col;
    const Inst& in = work_inst(inst0, kp, w, col);
    p3_sed_bulk<LANES>(in, col, kp, tb, sm, nullptr, err);
  });
  if (err) atomicOr(kp.err, err);
}

/* p3_sed_wide_kernel of the FP32-bulk form */
template <int LANES, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 3 * LANES : LANES)
    p3_sed_bulk_wide_kernel(const Inst inst0, const KParams<float> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<float> tb;
  sed_tables(kp, tb);
  constexpr int kGroups = SPLIT ? 3 : 1;
  const int g = SPLIT ? int(threadIdx.x) / LANES : 0;
  GroupScratch* const gs = reinterpret_cast<GroupScratch*>(smem_raw);
  double* const sm = reinterpret_cast<double*>(smem_raw + kGroups * sizeof(GroupScratch)) +
                     size_t(g) * sed_slots<float>() * kp.sm_stride;
  int col;
  const Inst& in = work_inst(inst0, kp, int(blockIdx.x), col);
  p3_sed_bulk<LANES, SPLIT>(in, col, kp, tb, sm, gs + g, err);
  if (err) atomicOr(kp.err, err);
}

template <class TR, int LANES>
__global__ void __launch_bounds__(256) p3_part3_kernel(const Inst inst0, const KParams<TR> kp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t err = 0;
  Tabs<TR> tb;
  setup_tables<TR>(kp, false, smem_raw, tb, err);
  const int split = kp.part3_split;
  for_each_work(kp.wctr ? kp.wctr + 2 : nullptr, kp.nwork * split, kp.groups_per_block, [&](int w) {
    const int item = split == 1 ? w : w / split;
    int col;
    const Inst& in = work_inst(inst0, kp, item, col);
    p3_part3<TR, LANES>(in, col, kp, tb, kp.work ? kp.work[item].inst : 0, (w - item * split) * LANES, split * LANES,
                        err);
  });
  if (err) atomicOr(kp.err, err);
}

}  // namespace dev
}  // namespace p3x
