// Advection-dispersion (ADE) step of FLUXOS-OVERLAND for sm_100a, the form for
// launches with few units in flight: a block takes one unit and splits each
// cell's work over its warps.
//
// ADEsolver_calc.cpp:27-291 re-scales every concentration to the new depth
// (:47-73) and then sweeps the grid once in Gauss-Seidel order (:93-290):
// cell (ix, iy) uses the already-updated concentration and limited fluxes of
// (ix-1, iy) and (ix, iy-1). Only a wavefront reproduces that order exactly.
//
// Mapping. A unit is a strip of 30 rows of one solute at one step; a block
// works on one unit at a time. Lane t (< 30) stands for row ix0 + t, and at
// warp step tau for cell (ix0 + t, tau - t + 1), so every lane's west
// neighbour is the cell lane t-1 finished one warp step earlier. What bounds
// the sweep is the chain of dependent cells (NR + NC of them whatever the
// layout), so the block's warps split a cell's work by what it depends on:
//   * the carry warp does only what needs the cells to the west and south:
//     the two upwind face values that read them, the outflow limiter, the
//     update. West carries (updated c, limited flux pfe) move lane t-1 -> t
//     with a shuffle, south carries stay in registers;
//   * NP face warps form everything else ahead of it, one warp step each of
//     every round of NP: the record of each cell (add_meteo's dilution, the
//     re-scale of :47-73, stored volume, 1/h), then from the records of the
//     cell and its neighbours the dispersive fluxes, the face values that do
//     not read a carry, the limits and the bounds of :51-62. Both pass
//     through shared memory;
//   * the helper warp waits for the progress of the strips this unit depends
//     on and copies concentrations (cp.async, L2 only: other SMs write them
//     during the launch) and boundary columns into shared rings; the publisher
//     warp makes the carry warp's progress known. So no fence, poll or global
//     load sits in the chain.
// A strip alone takes 0.27 us (FP32) and 0.53 us (FP64) a warp step, 540 and
// 1,040 cycles; one warp that does all of it in turn (fx_ade.cu) 0.73 and 1.85
// us. The cell's dependent operations alone, on registers, measure 260 and 430
// cycles, with the two votes 290 and 500; the rest is shared reads and waits.
// Eight steps of eight strips, each unit on an SM of its own, take 0.50 and
// 0.64 us a warp step.
//
// Steps in flight: as in fx_ade.cu, step j+1 of a strip follows step j a few
// rounds behind on the same and the next strip, and add_meteo's dilution
// (common.cpp:226-234) is applied to each record as it is formed.
//
// Units are handed out by a counter (fx_ctl::ade_next) in an order that has
// every unit behind the ones it waits for (fx_unit_order.h, fx_batch.cu),
// so whichever blocks are resident hold the oldest unfinished units and
// never wait on a unit that no block has taken. Strips of one step hand over
// through a small boundary buffer (per column: updated c, pfe, re-scaled c
// of the strip's last row); every dependency is a progress counter tagged
// with the step number. Every wait is bounded and sets fx_ctl::error when it
// gives up.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "fx_common.cuh"
#include "fx_internal.h"
#include "fx_unit_order.h"

namespace fxchain {

constexpr int ROWS = 30;      // rows per strip (lanes 0..29 compute)
constexpr int NP = 4;         // face warps: a round is NP warp steps
constexpr int FACE0 = 3;      // the first of them; before them the carry, helper and publisher warps
constexpr int NTHREADS = 32 * (FACE0 + NP);
constexpr int CR = 8;         // rounds of concentrations in flight
constexpr int RECS = 4 * NP;  // record slots: a face warp reads its round's records (one step back to
                              // two ahead) while the next round's are written: 3 NP + 1 at least
constexpr int RS = 36;        // records of a slot: the lanes', one before and three after them
constexpr int KR = 2;         // rounds of face coefficients between the face warps and the carry warp
constexpr int BR = 8;         // rounds of boundary columns
constexpr long long SPIN_LIMIT = 1LL << 20;  // idle polls of the helper warp (about a second) before giving up
constexpr long long HOLD_SPIN_LIMIT = 1LL << 12;  // the same with fx_dev.ade_hold (a test of the timeout path)
constexpr int WAIT_LIMIT = 1 << 24;  // tries of a wait inside the block (each suspends for a while)

// A cell's flag word for the carry warp.
constexpr unsigned K_VALID = 1u;   // a cell of the grid that this lane updates
constexpr unsigned K_KEEP = 2u;    // the re-scaled value stays (no sweep, or the cell it stops short of)
constexpr unsigned K_DRY = 4u;     // concentration and fluxes 0 (:119-124)
constexpr unsigned K_EAST = 8u;    // the east face value reads the west cell (:160-163)
constexpr unsigned K_NORTH = 16u;  // the north face value reads the south cell (:206-209)
constexpr unsigned K_DIV = 32u;    // divide by the depth the general way (see div_by)
constexpr unsigned K_SOIL = 64u;   // the soil release adds to the stored value

// What the carry warp needs of a cell, formed by the face warps.
template <class T>
struct Coef {
  T b;      // re-scaled concentration
  T v0;     // stored volume / dt
  T e1;     // east face: .375 c(E)
  T q1;     // fe_1
  T p1;     // dispersive flux, or with no carry the whole flux
  T l1;     // its limit -c(E) h(E) area / dt
  T e2, q2, p2, l2;  // north face
  T h;      // depth the update divides by
  T y;      // 1 / h (FP64 correctly rounded, FP32 the approximate reciprocal)
  T cmax, cmin;  // bounds (lane 0: without the west cell)
  T soil;   // soil release into this solute
  unsigned fl;
};

// Shared state of a block: the rings between its warps.
template <class T>
struct Smem {
  static constexpr int CV = 16 / sizeof(T);  // values of a 16-byte group
  static constexpr int NG = sizeof(T);       // groups of a cell's coefficients: 16 values
  T coef[KR * NP][NG][32][CV];
  // the 16-byte aligned group of concentrations that holds the lane's cell
  T c[CR * NP][32][CV];
  // records of the lanes' cells (entry lane + 1): re-scaled c and depth, c
  // before the sweep and stored volume / dt; bit lane of `dry`: a dry cell
  T bh[RECS][RS][2], cv[RECS][RS][2];
  unsigned dry[RECS];
  // boundary columns: c, pfe, re-scaled c of the west strip's last row; the
  // last entry is the ghost row's: 0
  T bnd[BR * NP + 1][4];
  // mbarriers: a round's concentrations have landed; its coefficients are
  // written, are read; its boundary columns are loaded
  unsigned long long c_full[CR], k_full[KR], k_empty[KR], b_full[BR];
  unsigned long long tick;  // one phase a round of the carry warp: what an idle warp sleeps on
  int done;     // warp steps the carry warp has finished
  int c_taken;  // rounds of concentrations the face warps have read
  int abort;    // a wait gave up
  int unit;
  int jj, k, s;  // the one-domain form: the unit's step, solute and strip
  fx_unit_walk walk;
};

// The state fields of the sweep in precision T.
template <class T>
struct Fields;
template <>
struct Fields<double> {
  static __device__ __forceinline__ double* conc(const fx_dev& d) { return d.conc; }
  static __device__ __forceinline__ double* soil(const fx_dev& d) { return d.soil; }
};
template <>
struct Fields<float> {
  static __device__ __forceinline__ float* conc(const fx_dev& d) { return d.conc_f; }
  static __device__ __forceinline__ float* soil(const fx_dev& d) { return d.soil_f; }
};

// Division and square root: IEEE-rounded in FP64 (bit parity with the
// reference); in FP32 the approximate hardware reciprocal and square root
// (PTX rcp.approx / sqrt.approx) refined by one Newton step with fused
// multiply-adds, without the IEEE code paths.
__device__ __forceinline__ float trcp(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
__device__ __forceinline__ double tdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float tdiv(float a, float b) {
  const float r = trcp(b);
  const float q = a * r;
  return fmaf(fmaf(-b, q, a), r, q);
}
__device__ __forceinline__ double tsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ float tsqrt(float a) {
  float s, r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(a));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
  const float t = fmaf(fmaf(-s, s, a), 0.5f * r, s);
  return a > 0.0f ? t : s;
}

// a / b with y = 1 / b known, the same bits as tdiv(a, b).
// FP64 (y correctly rounded): two Newton corrections of a * y. The first
// leaves a faithful quotient, so by Markstein's theorem (IBM J. Res. Dev. 34,
// 1990; Muller et al., Handbook of Floating-Point Arithmetic, ch. 4) the second
// rounds correctly; it needs exact residuals, hence the ranges of a (div_far)
// and of b (div_ok), outside of which the caller divides. A chain pays 5
// operations instead of a division (48 instead of 112 cycles measured).
__device__ __forceinline__ bool div_ok(double b) {  // 2^-200 < b < 2^200
  return (b > 6.223015277861142e-61) & (b < 1.6069380442589903e60);
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  const double q = fma(fma(-b, q1, a), y, q1);
  return a == 0.0 ? q0 : q;  // keeps the sign of 0
}
__device__ __forceinline__ bool div_far(double a) {  // |a| outside [2^-700, 2^700), and not 0
  const unsigned e = (unsigned)(__double2hiint(a) & 0x7ff00000) - ((1023u - 700u) << 20);
  return (e >= (1400u << 20)) & (a != 0.0);
}
__device__ __forceinline__ float div_by(float a, float b, float y) {
  const float q = a * y;
  return fmaf(fmaf(-b, q, a), y, q);
}
__device__ __forceinline__ bool div_far(float) { return false; }

// fmax and fmin (a NaN loses) as compares and selects: in FP64 half the
// instructions and latency of the functions.
__device__ __forceinline__ double tmax(double a, double b) { return (a > b) | (b != b) ? a : b; }
__device__ __forceinline__ double tmin(double a, double b) { return (a < b) | (b != b) ? a : b; }
__device__ __forceinline__ float tmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float tmin(float a, float b) { return fminf(a, b); }
// The same where b is no NaN.
__device__ __forceinline__ double pmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double pmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ float pmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float pmin(float a, float b) { return fminf(a, b); }

// The step a unit works on, in the sweep's precision, and the reciprocals its
// divisions share.
template <class T>
struct StepIn {
  long long cur;        // slot plane offset of the step
  double meteo_rate, dt64;
  T meteoi, mconc;
  T dt, y_dt;           // dt and its reciprocal (div_by)
  T dxy, area, D;
  T y_dxy, y_area;      // 1 / dxy and 1 / dxy^2: exact when dxy is a power of two (pow2)
  bool pow2;
  bool dt_ok;           // div_by may divide by dt
  long long inflow_gi;  // the point-inflow cell (-1: none)
  T inflow_add, inflow_hm;
  bool sweep;           // the sweep runs (hpall != 0 and it > 1)
  bool dilute;          // add_meteo's dilution runs
  bool melt;            // ... with a melt multiplier per cell (FP64)
  bool wintra;          // the soil release follows the sweep (hpall != 0)
};

__device__ __forceinline__ double recip(double b) { return 1.0 / b; }
__device__ __forceinline__ float recip(float b) { return trcp(b); }

template <class V>
__device__ __forceinline__ V shup(V v, int k) { return __shfl_up_sync(0xffffffffu, v, k); }

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Stores of the carry warp that no load of this thread depends on: without a
// memory clobber, so its shared loads of the next cell may pass them, and
// predicated, so its loop has no divergent branch.
__device__ __forceinline__ void put(bool on, double* p, double v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.global.f64 [%0], %1;\n}" ::"l"(p), "d"(v),
               "r"((unsigned)on));
}
__device__ __forceinline__ void put(bool on, float* p, float v) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.global.f32 [%0], %1;\n}" ::"l"(p), "f"(v),
               "r"((unsigned)on));
}
// Counters between the warps of a block.
__device__ __forceinline__ int ld_cta(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_cta(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Sleeps until the barrier's phase of this parity is over (true), a
// microsecond at most.
__device__ __forceinline__ bool mbar_doze(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(1000)
      : "memory");
  return ok != 0;
}
// Bounded wait for round `n` of a ring of R barriers (phase n / R of barrier
// n % R); false when it gave up or another warp did.
template <int R, class T>
__device__ __forceinline__ bool wait_round(Smem<T>& M, unsigned long long* bars, int n) {
  unsigned long long* bar = bars + n % R;
  const unsigned parity = (unsigned)(n / R) & 1u;
  if (mbar_try_wait(bar, parity)) return true;
  for (int k = 0; !mbar_try_wait(bar, parity); ++k) {
    if (ld_cta(&M.abort)) return false;
    if (k > WAIT_LIMIT) {
      st_cta(&M.abort, 1);
      return false;
    }
    if (k > 16) __nanosleep(200);
  }
  return true;
}
// Barrier of the face warps alone; true when any of their threads says so.
__device__ __forceinline__ bool face_sync_or(bool bad) {
  unsigned r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n barrier.cta.red.or.pred p, 1, %2, q;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(r)
      : "r"((unsigned)bad), "n"(NP * 32)
      : "memory");
  return r != 0;
}

// A cell's step inputs as loaded.
template <class T>
struct Raw {
  T h0, h, hp, mi, fe, fn;  // mi: FP32 the step's melt depth, FP64 the melt multiplier
  T fl;                     // a record's flag bits
  unsigned byte;            // the flag byte of a separate array
};

// A cell's record: what the unit's own cell keeps (its neighbours read b, c,
// h, v0 and the dry flag from shared memory).
template <class T>
struct Rec {
  T c;    // concentration before the sweep (after dilution, before re-scale)
  T b;    // re-scaled concentration (ADEsolver_calc.cpp:64-72)
  T h;    // depth after the hydrodynamic update
  T hd;   // the depth the update divides by (FP32: 1 in a cell without water)
  T y;    // its reciprocal
  T v0;   // (b * h) * area / dt
  T qx;   // fe_1 of the cell
  T qy;   // fn_1 of the cell
  T soil; // soil release into this solute
  unsigned fl;  // K_DRY, K_DIV, K_SOIL
};

// Loads the step inputs of the cell at plane element gi a round ahead of
// their use, straight into registers. No branch and no select stands behind
// the loads (either would wait for them): a lane whose cell is outside the
// grid is given another cell's element and does not use what it reads. The
// warp's lanes sit on 32 columns, so a record is one (FP32: 32 bytes) or two
// (FP64: 48 bytes) sectors of its own.
template <class T>
__device__ __forceinline__ void load_raw(const fx_dev& d, const StepIn<T>& S, long long gi, Raw<T>& r) {
  const long long o = S.cur + gi;
  if constexpr (sizeof(T) == 4) {
    const float4* p = d.rec32 + 2 * o;
    const float4 a = __ldg(p), b = __ldg(p + 1);
    r.h0 = a.x;
    r.h = a.y;
    r.hp = a.z;
    r.mi = a.w;
    r.fe = b.x;
    r.fn = b.y;
    r.fl = b.z;
  } else if (d.rec64) {  // a context
    const double2* p = reinterpret_cast<const double2*>(fx_rec64(d, o));
    const double2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    r.h0 = a.x;
    r.h = a.y;
    r.hp = b.x;
    r.fe = b.y;
    r.fn = c.x;
    r.fl = c.y;
    if (S.melt) r.mi = __ldg(d.melt_mult + gi);
  } else {  // fx_adesolver_noalloc: the caller's arrays (no melt, no slots)
    r.h0 = __ldg(d.h0 + o);
    r.h = __ldg(d.h + o);
    r.fe = __ldg(d.fe1 + o);
    r.fn = __ldg(d.fn1 + o);
    r.byte = __ldg(d.flags + o);
  }
}
// The flag byte of what was loaded.
__device__ __forceinline__ unsigned flags_of(const fx_dev&, const Raw<float>& r) { return __float_as_uint(r.fl); }
__device__ __forceinline__ unsigned flags_of(const fx_dev& d, const Raw<double>& r) {
  return d.rec64 ? (unsigned)__double2loint(r.fl) : r.byte;
}

// wintrasolver_calc (WINTRAsolver_calc.cpp:39-57) at one cell, for solute k:
// a wet cell whose bed is not NODATA_VALUE releases soil * rate / 3600 * dt
// of its soil mass into the concentration, c + deltam / (h * arbase), after
// the sweep. The reference calls it once per solute on one soil grid
// (main.cpp:400-404); this solute's copy of the soil mass replays every
// solute's release and keeps its own term. Nothing of it reads the swept
// concentration, so the face warps form the addend. The soil mass is read
// through L2 (other SMs wrote it in earlier steps).
template <class T>
__device__ __forceinline__ T soil_release(const fx_dev& d, const StepIn<T>& S, int k, long long gi, T h) {
  T* p = Fields<T>::soil(d) + (long long)k * d.plane + gi;
  T soil = __ldcg(p);
  T mine = T(0);
  for (int j = 0; j < d.nchem; ++j) {
    const T dm = tdiv(soil * (T)d.soil_rate, T(3600)) * S.dt;
    soil = soil - dm;
    if (j == k) mine = dm;
  }
  *p = soil;
  return tdiv(mine, h * (T)d.arbase);
}

// The record of a cell: add_meteo's dilution (common.cpp:214-234) when the
// step has one, then the re-scale of ADEsolver_calc.cpp:64-72 when the step
// sweeps. Ghost cells carry only their depth (their concentration is 0 and
// never changes). `cin` is the concentration as loaded; `in`: a cell of the
// grid, `interior`: no ghost cell; `release`: this lane updates the cell, and so its soil mass. Per-cell
// tests are selects; divisions that div_by cannot do are done again for the
// warp when one of its cells has one.
template <class T>
__device__ __forceinline__ Rec<T> make_rec(const fx_dev& d, const StepIn<T>& S, const Raw<T>& w, T cin, int k, bool in,
                                           bool interior, bool release, long long gi) {
  Rec<T> r;
  const unsigned fl = flags_of(d, w);
  const bool dry = fl & FX_F_LDRY, was_dry = fl & FX_F_LDRY_PREV;
  const T h = in ? w.h : T(0);
  const bool wet2 = !dry & !was_dry;  // wet before and after the step
  T c = interior ? cin : T(0);
  // the inflow cell holds h0 only after its inflow; the melt's dilution
  // divides by the depth after the melt (common.cpp:226-234, 313-325)
  const bool inflow_cell = gi == S.inflow_gi;
  const T hm = inflow_cell ? S.inflow_hm : w.h0;
  if (S.dilute) {
    // melt leaves hm >= hp > 0, evaporation may leave no depth: 0 / 0 then
    const bool use = interior & !(fl & FX_F_NODATA) & (w.hp != T(0));
    // the melt depth the hydrodynamic step added (fx_hydro.cu melt32, melt_depth)
    T mi = w.mi;
    if constexpr (sizeof(T) == 8) {
      mi = S.meteoi;
      if (d.melt_mult) {
        constexpr double day = 1000. * 3600. * 24.;
        const double rate = (double)S.meteo_rate * (double)w.mi;
        double q = div_by(rate, day, 1.0 / day);
        if (__any_sync(0xffffffffu, div_far(rate))) q = rate / day;
        mi = (T)(q * S.dt64);
      }
    }
    const T m = c * w.hp + (mi * S.mconc);
    // an FP64 division of 0 takes the long way; in FP32 0 over a subnormal depth is NaN (trcp)
    const bool some = use & ((sizeof(T) == 4) | (m != T(0)) | !(hm > T(0)));
    const T cd = tdiv(some ? m : T(1), some ? hm : T(1));
    c = some ? cd : (use ? m : c);
  }
  if (S.inflow_gi >= 0 && inflow_cell && interior && hm != T(0))
    c = tdiv(c * hm + S.inflow_add, w.h0);
  r.c = c;
  r.h = h;
  r.fl = dry & interior ? K_DRY : 0u;
  bool far;
  T b, v0;
  const T ch = c * w.h0;
  if constexpr (sizeof(T) == 4) {
    r.hd = h != T(0) ? h : T(1);
    far = false;
  } else {
    r.hd = div_ok(h) ? h : T(1);
    const bool ok = div_ok(h);
    r.fl |= !ok & !dry & interior ? K_DIV : 0u;
    far = interior & wet2 & (div_far(ch) | !ok);
  }
  r.y = recip(r.hd);
  T bw = div_by(ch, r.hd, r.y);
  // a threshold of 0 leaves cells wet without water; their quotient is NaN
  if constexpr (sizeof(T) == 4) bw = h != T(0) ? bw : __int_as_float(0x7fffffff);
  b = wet2 ? bw : (dry ? T(0) : c);
  b = S.sweep ? b : c;
  T vol = (b * h) * S.area;
  v0 = div_by(vol, S.dt, S.y_dt);
  if constexpr (sizeof(T) == 8) {
    if (__any_sync(0xffffffffu, far | !S.dt_ok | (interior & div_far(vol)))) {
      if (S.sweep && wet2) b = ch / h;
      vol = (b * h) * S.area;
      v0 = vol / S.dt;
    }
    r.hd = h;
  }
  r.b = interior ? b : T(0);
  r.v0 = interior ? v0 : T(0) * h;  // of a ghost cell 0, or NaN with no number for its depth
  r.qx = w.fe;
  r.qy = w.fn;
  r.soil = T(0);
  if (S.wintra && release && (double)h > d.hdry && !(fl & FX_F_NODATA)) {
    r.soil = soil_release<T>(d, S, k, gi, h);
    r.fl |= K_SOIL;
  }
  return r;
}

// One face of the cell without its carry (:151-194, :198-241). With a face
// value that reads the upwind carry (returned): its terms e, q and the
// dispersive flux p; else q = 0 and p the flux itself, and for a cell that is
// not updated (`act` false) 0. `to` is the cell across the face, `two` the
// one after it (b), `back_dry` the carry cell's dry flag.
template <class T>
__device__ __forceinline__ bool face(const StepIn<T>& S, bool act, T h, T fp, T q, T h_to, T f_to, bool dry_to, T f_two,
                                     bool dry_two, bool back_dry, bool edge, T& e, T& q_out, T& p) {
  const T hnu = pmax(h * h_to, T(.0001));
  // sqrt / sigc / dx * dy * D; sigc = 0.5: /sigc is *2 exactly, and with a
  // power of two / dx * dy leaves the value as it is
  T hn = tsqrt(hnu) * T(2);
  if (!S.pow2) {
    T g = div_by(hn, S.dxy, S.y_dxy);
    if (__any_sync(0xffffffffu, div_far(hn))) g = tdiv(hn, S.dxy);
    hn = g * S.dxy;
  }
  hn = hn * S.D;
  const T disp = dry_to ? T(0) : -hn * (f_to - fp);
  e = T(.375) * f_to;
  const bool down = q > T(0);
  const bool carry = act & !dry_to & down & !back_dry & !edge;
  const T mid = T(.5) * fp + T(.5) * f_to;
  const T dn = T(.375) * fp + T(.75) * f_to - T(.125) * f_two;
  T f = pmax((down | dry_two) ? mid : dn, T(0));
  f = (dry_to | edge) ? T(0) : f;  // :176-178, :223-225: the ghost concentration is 0
  const T whole = q * f * S.dxy + disp;
  p = act ? (carry ? disp : whole) : T(0);
  q_out = carry ? q : T(0);
  return carry;
}

// The coefficients of a lane's cell at warp step tau from its record and the
// records of its neighbours.
template <class T>
__device__ __forceinline__ Coef<T> make_coef(const StepIn<T>& S, const Smem<T>& M, const Rec<T>& r, int tau, int lane,
                                             bool valid, bool last_row, bool last_col, bool west_dry) {
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  Coef<T> k;
  const int sw = (tau - 1) & (RECS - 1), s1 = (tau + 1) & (RECS - 1), s2 = (tau + 2) & (RECS - 1);
  const V* rw = reinterpret_cast<const V*>(&M.bh[sw][lane][0]);
  const V* r1 = reinterpret_cast<const V*>(&M.bh[s1][lane][0]);
  const V* r2 = reinterpret_cast<const V*>(&M.bh[s2][lane][0]);
  const V* v1 = reinterpret_cast<const V*>(&M.cv[s1][lane][0]);
  const T Wb = rw[0].x, Sb = rw[1].x, NN = r2[1].x, EE = r2[3].x;
  const V N = r1[1], E = r1[2], Nc = v1[1], Ec = v1[2];
  const unsigned yw = (M.dry[sw] << 1) >> lane, y1 = M.dry[s1] >> lane, y2 = M.dry[s2] >> lane;
  const bool dW = lane == 0 ? west_dry : (yw & 1u), dS = yw & 2u, dN = y1 & 1u, dE = y1 & 2u;
  const T EEb = last_row ? E.x : EE, NNb = last_col ? N.x : NN;  // iee = min(ix+2, NROWS+1), inn alike
  const bool dEE = last_row ? dE : (y2 & 4u), dNN = last_col ? dN : (y2 & 1u);
  const bool act = valid & !(r.fl & K_DRY);
  k.fl = r.fl | (valid ? K_VALID : 0u);
  k.fl |= !S.sweep | (last_row & last_col) ? K_KEEP : 0u;  // :93
  k.b = r.b;
  k.h = r.hd;
  k.y = r.y;
  k.v0 = r.v0;
  k.soil = r.soil;
  T cmax = tmax(tmax(Sb, Nc.x), Ec.x), cmin = tmin(tmin(Sb, Nc.x), Ec.x);
  cmax = lane > 0 ? tmax(cmax, Wb) : cmax;
  cmin = lane > 0 ? tmin(cmin, Wb) : cmin;
  k.cmax = act ? cmax : T(0);
  k.cmin = act ? cmin : T(0);
  if (face<T>(S, act, r.h, r.b, r.qx, E.y, E.x, dE, EEb, dEE, dW, last_row, k.e1, k.q1, k.p1)) k.fl |= K_EAST;
  if (face<T>(S, act, r.h, r.b, r.qy, N.y, N.x, dN, NNb, dNN, dS, last_col, k.e2, k.q2, k.p2)) k.fl |= K_NORTH;
  // an inflow across the face is limited by what the cell it leaves holds
  // (:187-194); across a dry face there is none
  k.l1 = dE ? T(0) : -Ec.y;
  k.l2 = dN ? T(0) : -Nc.y;
  return k;
}

__device__ __forceinline__ void put_coef(Smem<double>& M, int slot, int lane, const Coef<double>& k) {
  double2* p = reinterpret_cast<double2*>(&M.coef[slot][0][lane][0]);
  p[0] = make_double2(k.b, k.v0);
  p[32] = make_double2(k.e2, k.q2);
  p[64] = make_double2(k.p2, k.l2);
  p[96] = make_double2(k.e1, k.q1);
  p[128] = make_double2(k.p1, k.l1);
  p[160] = make_double2(k.h, k.y);
  p[192] = make_double2(k.cmax, k.cmin);
  p[224] = make_double2(__longlong_as_double((long long)k.fl), k.soil);
}
__device__ __forceinline__ void put_coef(Smem<float>& M, int slot, int lane, const Coef<float>& k) {
  float4* p = reinterpret_cast<float4*>(&M.coef[slot][0][lane][0]);
  p[0] = make_float4(k.b, k.v0, k.e2, k.q2);
  p[32] = make_float4(k.p2, k.l2, k.e1, k.q1);
  p[64] = make_float4(k.p1, k.l1, k.h, k.y);
  p[96] = make_float4(k.cmax, k.cmin, __uint_as_float(k.fl), k.soil);
}
__device__ __forceinline__ void get_coef(const Smem<double>& M, int slot, int lane, Coef<double>& k) {
  const double2* p = reinterpret_cast<const double2*>(&M.coef[slot][0][lane][0]);
  const double2 a = p[0], b = p[32], c = p[64], e = p[96], f = p[128], g = p[160], h = p[192], i = p[224];
  k = Coef<double>{a.x, a.y, e.x, e.y, f.x, f.y, b.x, b.y, c.x, c.y, g.x, g.y, h.x, h.y, i.y,
                   (unsigned)__double2loint(i.x)};
}
__device__ __forceinline__ void get_coef(const Smem<float>& M, int slot, int lane, Coef<float>& k) {
  const float4* p = reinterpret_cast<const float4*>(&M.coef[slot][0][lane][0]);
  const float4 a = p[0], b = p[32], c = p[64], e = p[96];
  k = Coef<float>{a.x, a.y, b.z, b.w, c.x, c.y, a.z, a.w, b.x, b.y, c.z, c.w, e.x, e.y, e.w, __float_as_uint(e.z)};
}

// The unit's part of the step: what its warps share.
template <class T>
struct Unit {
  StepIn<T> S;
  long long step;
  int slot, jj, k, s, nstrips, TW, rounds;
  int ix0;
};

// Fills `U` for strip s of solute k at the jj-th live step of the batch;
// false when the batch has fewer steps. Every warp does this for itself.
template <class T>
__device__ __forceinline__ bool open_unit(const fx_dev& d, Unit<T>& U, int jj, int k, int s, int lane) {
  const fx_ctl& cc = *d.ctl;
  // this batch's live steps are consecutive: the jj-th is minstep + jj
  int m = 0;
  long long minstep = 0x7fffffffffffffffLL;
  for (int q0 = 0; q0 < d.nslot; q0 += 32) {
    const int q = q0 + lane;
    bool mine = false;
    if (q < d.nslot) {
      const fx_steprec& r = cc.rec[q];
      mine = r.live && r.batch == cc.batch;
      if (mine) minstep = min(minstep, r.step);
    }
    m += __popc(__ballot_sync(0xffffffffu, mine));
  }
  if (jj >= m) return false;
  for (int o = 16; o > 0; o >>= 1) minstep = min(minstep, __shfl_xor_sync(0xffffffffu, minstep, o));
  U.step = minstep + jj;
  U.slot = (int)(U.step % d.nslot);
  U.jj = jj;
  U.k = k;
  U.s = s;
  U.nstrips = (d.nr + ROWS - 1) / ROWS;
  U.TW = d.nc + ROWS - 1;  // warp steps per strip
  U.rounds = (U.TW + NP - 1) / NP;
  U.ix0 = 1 + s * ROWS;
  const fx_steprec& rec = cc.rec[U.slot];
  StepIn<T>& S = U.S;
  S.cur = fx_slot(d, rec.step);
  S.meteo_rate = rec.meteo_rate;
  S.dt64 = rec.dtfl;
  S.meteoi = (T)rec.meteoi;
  S.mconc = (T)rec.mconc;
  S.dt = (T)rec.dtfl;
  S.y_dt = recip(S.dt);
  S.dxy = (T)d.dxy;
  S.area = (T)d.arbase;
  S.D = (T)d.dcoef[k];
  S.pow2 = d.dxy_pow2 != 0;
  S.y_dxy = recip(S.dxy);
  S.y_area = S.pow2 ? (T)d.inv_area : recip(S.area);
  S.dt_ok = div_ok((double)S.dt);
  S.sweep = rec.active && rec.it > 1;  // :45,74-77
  S.dilute = d.has_meteo != 0;
  S.melt = sizeof(T) == 8 && S.dilute && d.melt_mult;
  S.wintra = d.wintra && rec.active;  // main.cpp:385-405
  S.inflow_gi = d.has_inflow ? d.inflow_gi : -1;
  S.inflow_add = (T)(rec.inflowi * rec.iconc);
  S.inflow_hm = (T)rec.inflow_hm;
  return true;
}

// The flux limits of ADEsolver_calc.cpp:187-194, :234-241, the outflow limiter
// of :243-278 and the update of :281-288 in the general form, for any
// operands: fluxes before their limits in pfe, qfn (limited on return).
// inv_area: 1 / area where that is exact, else 0.
template <class T>
__device__ __noinline__ T cell_general(T v0, T W_pfe, T o_qfn, T l1, T l2, T dt, T area, T inv_area, T b, T h, T cmax, T cmin,
                                       T& pfe_io, T& qfn_io) {
  T pfe = pfe_io, qfn = qfn_io;
  if (pfe < T(0)) pfe = fmax(pfe, l1);
  if (qfn < T(0)) qfn = fmax(qfn, l2);
  const T have = v0 + W_pfe + o_qfn;
  if (have > T(0)) {
    if (pfe > T(0) && qfn > T(0)) {
      if (pfe + qfn > have) {
        const T cf = tdiv(qfn, pfe + qfn);
        pfe = (T(1) - cf) * have;
        qfn = cf * have;
      }
    } else if (pfe > T(0)) {
      pfe = fmin(pfe, (have - qfn));
    } else if (qfn > T(0)) {
      qfn = fmin(qfn, (have - pfe));
    }
  } else {
    if (pfe >= T(0) && qfn < T(0)) {
      const T left = have - qfn;
      pfe = left > T(0) ? fmin(pfe, left) : T(0);
    } else if (pfe < T(0) && qfn >= T(0)) {
      const T left = have - pfe;
      qfn = left > T(0) ? fmin(qfn, left) : T(0);
    } else if (pfe >= T(0) && qfn >= T(0)) {
      pfe = T(0);
      qfn = T(0);
    }
  }
  const T flux = (W_pfe - pfe + o_qfn - qfn) * dt;
  const T dc = inv_area != T(0) ? flux * inv_area : tdiv(flux, area);
  T cn = b + tdiv(dc, h);
  cn = fmin(cmax, cn);
  cn = fmax(cmin, cn);
  pfe_io = pfe;
  qfn_io = qfn;
  return cn;
}

// The carry warp: the unit's chain of dependent cells. Bound by the latency
// of one cell (about 30 dependent operations), so everything that can be
// known before the west and south cells is read ready-made from `coef`, and
// the cell is one straight-line block of selects. A cell that is not updated
// has coefficients that make its value and fluxes 0; a NaN, a quotient that
// div_by cannot form or a cell that keeps its value sends the warp through
// the general form for that warp step.
template <class T>
__device__ __forceinline__ bool carry_warp(const fx_dev& d, const Unit<T>& U, Smem<T>& M, int lane, int& k_round,
                                           int& b_round) {
  const int ix = U.ix0 + lane;
  // the lane's cell at warp step tau is column tau - lane + 1
  T* A = (T*)__cvta_generic_to_global(Fields<T>::conc(d) + U.k * d.plane) + fx_ix(d, ix, 1) - (long long)lane * d.ld;
  const bool hand = lane == ROWS - 1 && U.s + 1 < U.nstrips;
  double* bnd_out = (double*)__cvta_generic_to_global(d.ade_bnd) + (((long long)U.slot * d.nchem + U.k) * U.nstrips + U.s + (hand ? 1 : 0)) *
                                    ((long long)(d.nc + 2) * 3) - 3 * (lane - 1);
  const bool west = U.s > 0;
  // outputs of this lane's previous cell: its south cell for the next step,
  // its west cell for lane + 1
  T o_c = T(0), o_pfe = T(0), o_qfn = T(0);
  const T dt = U.S.dt, dxy = U.S.dxy, area = U.S.area, y_area = U.S.y_area;
  const bool pow2 = U.S.pow2, wintra = U.S.wintra, sweep = U.S.sweep;
  const long long ld = d.ld;
  for (int q = 0; q < U.rounds; ++q, ++k_round) {
    if (!wait_round<KR>(M, M.k_full, k_round)) return false;
    if (west && !wait_round<BR>(M, M.b_full, b_round)) return false;
    Coef<T> next;
    // the west strip's last row, or the ghost row 0: c = 0 and pfe = the
    // ghost convective flux c(0,iy)*fe_1(0,iy)*dy = 0 (:106-116)
    const T* bw = M.bnd[west ? (b_round % BR) * NP : BR * NP];
    const int bstep = west ? 4 : 0;
    get_coef(M, (k_round % KR) * NP, lane, next);
    T n_c = bw[0], n_pfe = bw[1], n_b = bw[2];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const Coef<T> c = next;
      const T t_c = n_c, t_pfe = n_pfe, t_b = n_b;
      T W_c = shup(o_c, 1), W_pfe = shup(o_pfe, 1);
      if (i + 1 < NP) {
        get_coef(M, (k_round % KR) * NP + i + 1, lane, next);
        n_c = bw[(i + 1) * bstep];
        n_pfe = bw[(i + 1) * bstep + 1];
        n_b = bw[(i + 1) * bstep + 2];
      }
      // The expressions of ADEsolver_calc.cpp:126-288 in the same order
      // and operand types; both sides of every test are evaluated and the
      // result selected. The north face first: it needs no neighbour lane.
      const T p75 = T(.75) * c.b;
      const T fn = pmax(T(-.125) * o_c + p75 + c.e2, T(0));
      const T qfn0 = c.q2 * fn * dxy + c.p2;
      const T qfn = qfn0 < T(0) ? pmax(qfn0, c.l2) : qfn0;
      const bool edge = (lane == 0) & !(c.fl & K_DRY);
      const T wb1 = edge ? t_b : c.cmax, wb2 = edge ? t_b : c.cmin;
      const T cmax = pmax(wb1, c.cmax), cmin = pmin(wb2, c.cmin);
      W_c = lane == 0 ? t_c : W_c;
      W_pfe = lane == 0 ? t_pfe : W_pfe;
      const T fe = pmax(T(-.125) * W_c + p75 + c.e1, T(0));
      const T pfe0 = c.q1 * fe * dxy + c.p1;
      const T pfe = pfe0 < T(0) ? pmax(pfe0, c.l1) : pfe0;
      // outflow limiter (:243-278)
      const T have = c.v0 + W_pfe + o_qfn;
      const T sum = pfe + qfn;
      const bool pos = have > T(0);
      const bool pp = pfe > T(0), qp = qfn > T(0), pn = pfe < T(0), qn = qfn < T(0);
      const T m1 = have - qfn, m2 = have - pfe;
      // have > 0: the only outflow takes at most what is left; have <= 0:
      // an outflow beside an inflow likewise, at least 0, and without one none
      // (bitwise logic: && and || would become branches)
      const bool use1 = (pos & pp & !qp) | (!pos & !pn & qn), use2 = (pos & qp & !pp) | (!pos & pn & !qn);
      const bool none = !pos & !pn & !qn;
      const bool zero1 = none | (use1 & !pos & !(m1 > T(0))), zero2 = none | (use2 & !pos & !(m2 > T(0)));
      const T f1 = pmin(pfe, m1), f2 = pmin(qfn, m2);
      T pl = use1 ? f1 : pfe;
      T ql = use2 ? f2 : qfn;
      pl = zero1 ? T(0) : pl;
      ql = zero2 ? T(0) : ql;
      const bool split = pos & pp & qp & (sum > have);
      // two outflows share what is there (a division, when a lane needs it)
      if (__any_sync(0xffffffffu, split)) {
        const T cf = tdiv(split ? qfn : T(1), split ? sum : T(1));
        pl = split ? (T(1) - cf) * have : pl;
        ql = split ? cf * have : ql;
      }
      const T flux = (W_pfe - pl + o_qfn - ql) * dt;  // :281-286
      const T dc = pow2 ? flux * y_area : div_by(flux, area, y_area);
      T cn = c.b + div_by(dc, c.h, c.y);
      cn = pmin(cmax, cn);
      cn = pmax(cn, cmin);
      // (FP32 minima and maxima are the general form's, so cmax may be a NaN)
      const T nan = sizeof(T) == 8 ? sum + have + cmax : sum + have;
      bool odd = c.fl & (K_DIV | K_KEEP);
      odd = odd | !(nan == nan) | div_far(dc) | (!pow2 & div_far(flux));
      if (__any_sync(0xffffffffu, odd)) {
        const bool flow = (c.fl & (K_KEEP | K_DRY | K_VALID)) == K_VALID;
        T g = T(0), gp = (c.fl & K_EAST) ? pfe0 : c.p1, gq = (c.fl & K_NORTH) ? qfn0 : c.p2;
        if (sweep)  // a step without one keeps every cell (700 x 700, two solutes, FP64 1.06 ms; 2.67 with the call)
          g = cell_general<T>(c.v0, W_pfe, o_qfn, c.l1, c.l2, dt, area, pow2 ? y_area : T(0), c.b, c.h,
                              fmax(wb1, c.cmax), fmin(wb2, c.cmin), gp, gq);
        cn = flow ? g : ((c.fl & K_KEEP) ? c.b : T(0));
        pl = flow ? gp : T(0);
        ql = flow ? gq : T(0);
      }
      // the sweep's neighbours and the next strip read the value before the
      // soil release, which follows the whole sweep in the reference
      const bool valid = c.fl & K_VALID;
      put(valid, A, wintra & ((c.fl & K_SOIL) != 0) ? cn + c.soil : cn);
      const bool give = valid & hand;
      put(give, bnd_out, (double)cn);
      put(give, bnd_out + 1, (double)pl);
      put(give, bnd_out + 2, (double)c.b);
      o_c = cn;
      o_pfe = pl;
      o_qfn = ql;
      A += ld;
      bnd_out += 3;
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&M.k_empty[k_round % KR]);
      mbar_arrive(&M.tick);
      st_cta(&M.done, min((q + 1) * NP, U.TW));
    }
    if (west) ++b_round;
  }
  return true;
}

// A face warp: the records of its warp steps (one per round), then, when the
// round's records are in shared memory, the coefficients of its warp step of
// the round before. Bound by instruction issue; its step inputs are loaded
// a round ahead into registers (two sets, used in turn: a copy between them
// would wait for the loads).
template <class T>
__device__ __forceinline__ bool face_warp(const fx_dev& d, const Unit<T>& U, Smem<T>& M, int p, int lane, int& c_round,
                                          int& k_round) {
  const StepIn<T>& S = U.S;
  const int ix = U.ix0 + lane;
  const bool row_in = ix <= d.nr + 1, row_int = ix <= d.nr, last_row = ix == d.nr, mine = row_int && lane < ROWS;
  const unsigned nc = (unsigned)d.nc;
  bool bad = false;
  int iy = p - lane + 1;  // this lane's column in round 0
  const long long ahead = (long long)NP * d.ld;
  long long gi = fx_ix(d, ix, iy);  // read for columns of the grid only
  // the dry flag of the west strip's last row, for lane 0
  const bool west0 = U.s > 0 && lane == 0;
  struct In {
    Raw<T> w;
    unsigned west;
    Rec<T> rec;
  };
  auto load = [&](In& x, int col, long long g) {
    load_raw<T>(d, S, row_in && (unsigned)col <= nc + 1 ? g : 0, x.w);
    if (west0 && (unsigned)(col - 1) < nc) x.west = __ldg(d.flags + S.cur + g - 1);
  };
  // round r with its inputs in x: records; coefficients of the round before,
  // whose record is in y, and y takes the inputs of the next round
  auto round = [&](int r, In& x, In& y) -> bool {
    const Rec<T> own = y.rec;
    const bool own_west_dry = y.west & FX_F_LDRY;
    load(y, iy + NP, gi + ahead);
    if (!wait_round<CR>(M, M.c_full, c_round)) bad = true;
    const bool interior = row_int && (unsigned)(iy - 1) < nc;
    const T cin = M.c[(c_round % CR) * NP + p][lane][(int)gi & (Smem<T>::CV - 1)];
    x.rec = make_rec<T>(d, S, x.w, cin, U.k, row_in && (unsigned)iy <= nc + 1, interior, interior && lane < ROWS && !bad, gi);
    const int rho = r * NP + p, slot = rho & (RECS - 1);
    M.bh[slot][lane + 1][0] = x.rec.b;
    M.bh[slot][lane + 1][1] = x.rec.h;
    M.cv[slot][lane + 1][0] = x.rec.c;
    M.cv[slot][lane + 1][1] = x.rec.v0;
    const unsigned dry = __ballot_sync(0xffffffffu, x.rec.fl & K_DRY);
    if (lane == 0) M.dry[slot] = dry;
    if (face_sync_or(bad)) return false;
    if (p == 0 && lane == 0) st_cta(&M.c_taken, r + 1);
    if (r > 0) {
      const int col = iy - NP;
      const Coef<T> k = make_coef<T>(S, M, own, rho - NP, lane, mine && (unsigned)(col - 1) < nc, last_row, col == (int)nc,
                                     own_west_dry);
      // the slot's last user is KR rounds back: its phase before this one
      if (k_round < KR || wait_round<KR>(M, M.k_empty, k_round - KR)) {
        put_coef(M, (k_round % KR) * NP + p, lane, k);
        __syncwarp();
        if (lane == 0) mbar_arrive(&M.k_full[k_round % KR]);
      } else {
        bad = true;
      }
      ++k_round;
    }
    ++c_round;
    iy += NP;
    gi += ahead;
    return true;
  };
  In a, b;
  a.west = b.west = 0u;
  a.w.h0 = a.w.h = a.w.hp = a.w.mi = a.w.fe = a.w.fn = a.w.fl = T(0);
  a.w.byte = 0u;
  b.w = a.w;
  load(a, iy, gi);
  b.rec.fl = 0;
  for (int r = 0; r <= U.rounds; r += 2) {
    if (!round(r, a, b)) return false;
    if (r < U.rounds && !round(r + 1, b, a)) return false;
  }
  return !bad;
}

// A count of warp steps of a strip whose counter holds (step << 32 | count).
__device__ __forceinline__ int count_of(unsigned long long v, unsigned long long tag) {
  const unsigned t = (unsigned)(v >> 32), want = (unsigned)tag;
  return t == want ? (int)(unsigned)v : (t > want ? 0x7fffffff : -1);
}

// The helper warp: dependencies and copies in. With d.ade_hold set
// (fx_set_option "fail_ade_waits") a unit that has a dependency never sees it
// met, so its wait runs out after HOLD_SPIN_LIMIT polls: the timeout path,
// exercised without a fault.
template <class T>
__device__ __forceinline__ bool helper_warp(const fx_dev& d, const Unit<T>& U, Smem<T>& M, int lane, int& c_round,
                                            int& b_round) {
  const T* A = Fields<T>::conc(d) + U.k * d.plane;
  auto unit_index = [&](int sl, int ss) { return ((long long)sl * d.nchem + U.k) * U.nstrips + ss; };
  const unsigned long long tag = (unsigned long long)U.step;
  const int pslot = (int)((U.step - 1) % d.nslot);
  const double* bnd_in = d.ade_bnd + unit_index(U.slot, U.s) * ((long long)(d.nc + 2) * 3);
  // the three counters the unit depends on, one per lane: the west strip of
  // this step and, on the previous step of the batch (earlier batches are
  // complete), this strip and the next one
  const bool west = U.s > 0, prev0 = U.jj > 0, prev1 = U.jj > 0 && U.s + 1 < U.nstrips;
  const unsigned long long* mine = nullptr;
  if (lane == 0 && west) mine = d.ade_prog + unit_index(U.slot, U.s - 1);
  if (lane == 1 && prev0) mine = d.ade_prog + unit_index(pslot, U.s);
  if (lane == 2 && prev1) mine = d.ade_prog + unit_index(pslot, U.s + 1);
  const bool hold = d.ade_hold != 0 && (west || prev0 || prev1);
  const long long limit = hold ? HOLD_SPIN_LIMIT : SPIN_LIMIT;
  // counts seen; a dependency the unit does not have is met from the start
  int seen_w = west ? -1 : 0x7fffffff, seen_p0 = prev0 ? -1 : 0x7fffffff, seen_p1 = prev1 ? -1 : 0x7fffffff;
  // Round r's concentrations are read at warp steps r*NP .. r*NP + NP-1. Lane
  // t < ROWS reads its row at the column that the previous step's sweep of
  // this strip, on the same skew, updates at the same warp step; lanes ROWS
  // and ROWS + 1 read the next strip's rows 0 and 1, at columns that strip's
  // lanes 0 and 1 update ROWS - 1 warp steps earlier. Round q's boundary
  // columns end at q*NP + NP, which the west strip's lane ROWS - 1 updates
  // ROWS - 1 warp steps later than its lane 0. (Each strip also writes its
  // own cells only after the previous step did, and the next strip's first
  // rows are overwritten by its own sweep only ROWS warp steps behind this
  // strip's, after this strip has read them; these counts cover both.)
  auto need_p0 = [&](int r) { return min(r * NP + NP, U.TW); };
  auto need_p1 = [&](int r) { return max(0, min(r * NP + NP - ROWS, U.TW)); };
  auto need_w = [&](int q) { return min(q * NP + NP + ROWS - 1, U.TW); };
  const int c_rounds = U.rounds + 1, b_rounds = west ? U.rounds : 0;
  const int ix = U.ix0 + lane;
  const bool row_int = ix <= d.nr;
  int iy = 1 - lane;                // this lane's column at the next warp step to copy
  long long gi = fx_ix(d, ix, iy);  // read for columns of the grid only
  int rc = 0, qb = 0;
  unsigned tick = 0;
  long long idle = 0;
  while (rc < c_rounds || qb < b_rounds) {
    bool moved = false;
    const bool want_c = rc < c_rounds && (seen_p0 < need_p0(rc) || seen_p1 < need_p1(rc));
    const bool want_w = qb < b_rounds && seen_w < need_w(qb);
    if (want_c || want_w) {
      // the counters in one round trip
      const unsigned long long v = mine ? ld_relaxed(mine) : 0ull;
      const unsigned long long want_tag = lane == 0 ? tag : tag - 1;
      int n = mine ? count_of(v, want_tag) : 0x7fffffff;
      const int had = lane == 0 ? seen_w : (lane == 1 ? seen_p0 : seen_p1);
      if (__any_sync(0xffffffffu, mine && n > had)) {
        // read again with acquire: it and the warp barrier order the lanes'
        // later reads of the producers' data after the counts. (A poll that
        // sees nothing new stays relaxed: an acquire empties the SM's L1.)
        if (mine) n = count_of(ld_acquire(mine), want_tag);
        seen_w = __shfl_sync(0xffffffffu, n, 0);
        seen_p0 = __shfl_sync(0xffffffffu, n, 1);
        seen_p1 = __shfl_sync(0xffffffffu, n, 2);
        __syncwarp();
      }
    }
    if (!hold) {
      if (qb < b_rounds) {
        // boundary columns of as many rounds as the ring and the west strip allow
        const int room = min(b_rounds, ld_cta(&M.done) / NP + BR);
        int n = 0;
        while (n < BR && qb + n < room && seen_w >= need_w(qb + n)) ++n;
        if (n > 0) {
          static_assert(BR * NP <= 32, "a lane per boundary column");
          const int col = qb * NP + lane + 1;
          if (lane < n * NP) {
            T v0 = T(0), v1 = T(0), v2 = T(0);
            if (col <= d.nc) {
              const double* p = bnd_in + (long long)col * 3;
              v0 = (T)__ldcg(p);
              v1 = (T)__ldcg(p + 1);
              v2 = (T)__ldcg(p + 2);
            }
            T* t = M.bnd[(b_round * NP + lane) % (BR * NP)];
            t[0] = v0;
            t[1] = v1;
            t[2] = v2;
          }
          __syncwarp();
          if (lane < n) mbar_arrive(&M.b_full[(b_round + lane) % BR]);
          qb += n;
          b_round += n;
          moved = true;
        }
      }
      const int room = min(c_rounds, ld_cta(&M.c_taken) + CR);
      while (rc < room && seen_p0 >= need_p0(rc) && seen_p1 >= need_p1(rc)) {
        const int cs = c_round % CR;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          if (row_int && (unsigned)(iy - 1) < (unsigned)d.nc)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&M.c[cs * NP + i][lane][0])),
                         "l"(__cvta_generic_to_global(A + (gi & ~(long long)(Smem<T>::CV - 1))))
                         : "memory");
          ++iy;
          gi += d.ld;
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&M.c_full[cs])) : "memory");
        ++rc;
        ++c_round;
        moved = true;
      }
    }
    if (moved) {
      idle = 0;
      continue;
    }
    const bool stop = ++idle > limit || ld_cta(&M.abort) != 0 ||
                      ((idle & 63) == 0 && *(volatile int*)&d.ctl->error != 0);
    if (__any_sync(0xffffffffu, stop)) return false;
    if (want_c || want_w) __nanosleep(idle < 1024 ? 200 : 500);  // other blocks' progress
    else if (mbar_doze(&M.tick, tick)) tick ^= 1u;               // room in a ring: a round of this block
  }
  return true;
}

// The publisher warp: makes the carry warp's progress known to the strips
// that depend on this one. The carry warp's writes are ordered before its
// count in shared memory, and by the fence before the count published here;
// the fence takes about as long as a round, so it has a warp of its own.
template <class T>
__device__ __forceinline__ bool publisher_warp(const fx_dev& d, const Unit<T>& U, Smem<T>& M) {
  unsigned long long* prog = d.ade_prog + ((long long)U.slot * d.nchem + U.k) * U.nstrips + U.s;
  const unsigned long long tag = (unsigned long long)U.step << 32;
  int published = 0;
  unsigned tick = 0;
  // its bound is the other warps': they set `abort` when a wait gives up
  for (long long idle = 0; published < U.TW;) {
    const int done = ld_cta(&M.done);
    if (done > published) {
      if ((threadIdx.x & 31) == 0) st_release(prog, tag | (unsigned)done);
      published = done;
      idle = 0;
      continue;
    }
    if (ld_cta(&M.abort) || ++idle > 8 * SPIN_LIMIT) return false;
    if (mbar_doze(&M.tick, tick)) tick ^= 1u;
  }
  return true;
}

// One unit by the block's warps. `c_round`, `k_round` and `b_round` count the
// rounds of concentrations, coefficients and boundary columns since the
// launch (the phases of the rings' barriers).
template <class T>
__device__ __forceinline__ void run_unit(const fx_dev& d, Smem<T>& M, int jj, int k, int s, int& c_round, int& k_round,
                                         int& b_round) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Unit<T> U;
  if (!open_unit<T>(d, U, jj, k, s, lane)) return;
  bool ok;
  if (warp == 0) ok = carry_warp<T>(d, U, M, lane, k_round, b_round);
  else if (warp == 1) ok = helper_warp<T>(d, U, M, lane, c_round, b_round);
  else if (warp == 2) ok = publisher_warp<T>(d, U, M);
  else ok = face_warp<T>(d, U, M, warp - FACE0, lane, c_round, k_round);
  if (!ok) {
    st_cta(&M.abort, 1);
    if (lane == 0) atomicCAS(&d.ctl->error, 0, FX_DEVERR_WAIT_TIMEOUT);
  }
}

template <class T>
__device__ __forceinline__ void init_smem(Smem<T>& M) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < CR; ++i) mbar_init(&M.c_full[i], 32);
    for (int i = 0; i < KR; ++i) mbar_init(&M.k_full[i], NP);
    for (int i = 0; i < KR; ++i) mbar_init(&M.k_empty[i], 1);
    for (int i = 0; i < BR; ++i) mbar_init(&M.b_full[i], 1);
    mbar_init(&M.tick, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    M.abort = 0;
    for (int i = 0; i < 4; ++i) M.bnd[BR * NP][i] = T(0);
  }
  // entries beyond the lanes' own, read by lanes that update no cell
  for (int k = threadIdx.x; k < RECS * RS; k += NTHREADS) {
    const int e = k % RS;
    if (e == 0 || e > 32)
      for (int v = 0; v < 2; ++v) M.bh[k / RS][e][v] = M.cv[k / RS][e][v] = T(0);
  }
}

// Takes the block's next unit (every thread calls it); -1 when there is none
// or a wait gave up.
// `decode` is called with it by the thread that took it.
template <class T, class F>
__device__ __forceinline__ int next_unit(Smem<T>& M, int* counter, int nunits, F decode) {
  __syncthreads();  // every warp is done with the last unit
  if (threadIdx.x == 0) {
    const int u = atomicAdd(counter, 1);
    M.unit = (u < nunits && !M.abort) ? u : -1;
    M.done = M.c_taken = 0;
    if (M.unit >= 0) decode(M.unit);
  }
  // what the first warp step finds to its west and south: the ghost cells
  if (threadIdx.x < RS) M.bh[RECS - 1][threadIdx.x][0] = M.bh[RECS - 1][threadIdx.x][1] = T(0);
  if (threadIdx.x == 0) M.dry[RECS - 1] = 0;
  __syncthreads();
  return M.unit;
}

// Resident blocks per SM the kernels are compiled for: 2 x 7 warps at 128
// registers (FP64), 3 x 7 at 80 (FP32). One block less is 8 to 20 % faster
// where a block per SM is enough and 18 to 20 % slower at 1,000 x 700 cells
// and more; one block more spills (1,000 x 700 FP64 0.187 -> 0.249 ms a step).
template <class T>
struct ChainBlocks {
  static constexpr int value = sizeof(T) == 8 ? 2 : 3;
};

// One domain: the descriptor is a kernel parameter. Unit u is solute
// u % nchem of the step and strip that fx_unit_at gives for u / nchem.
template <class T>
__global__ void __launch_bounds__(NTHREADS, ChainBlocks<T>::value) k_chain_one(const __grid_constant__ fx_dev d, int steps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<T>& M = *reinterpret_cast<Smem<T>*>(smem_raw);
  if (!d.ade) return;
  init_smem(M);
  const int nstrips = (d.nr + ROWS - 1) / ROWS;
  if (threadIdx.x == 0) M.walk = fx_unit_walk{0, 0};
  int c_round = 0, k_round = 0, b_round = 0;
  for (;;) {
    const int u = next_unit(M, &d.ctl->ade_next, steps * d.nchem * nstrips, [&](int i) {
      M.k = i % d.nchem;
      fx_unit_at(i / d.nchem, steps, nstrips, M.walk, M.jj, M.s);
    });
    if (u < 0) break;
    run_unit<T>(d, M, M.jj, M.k, M.s, c_round, k_round, b_round);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// A batch of domains: units come from the unit table; the block copies its
// unit's descriptor to shared memory. The first domain's control block holds
// the unit counter.
template <class T>
__global__ void __launch_bounds__(NTHREADS, ChainBlocks<T>::value) k_chain_batch(const fx_dev* __restrict__ devs,
                                                         const fx_unit* __restrict__ units, int nunits) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<T>& M = *reinterpret_cast<Smem<T>*>(smem_raw);
  __shared__ fx_dev sdev;
  init_smem(M);
  int have = -1, c_round = 0, k_round = 0, b_round = 0;
  int* counter = &devs[0].ctl->ade_next;
  for (;;) {
    const int u = next_unit(M, counter, nunits, [](int) {});
    if (u < 0) break;
    const fx_unit un = units[u];
    if (un.dom != have) {
      const unsigned long long* src = reinterpret_cast<const unsigned long long*>(devs + un.dom);
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sdev);
      for (int i = threadIdx.x; i < (int)(sizeof(fx_dev) / 8); i += NTHREADS) dst[i] = src[i];
      __syncthreads();
      have = un.dom;
    }
    if (!sdev.ade) continue;
    run_unit<T>(sdev, M, un.jj, un.k, un.s, c_round, k_round, b_round);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace fxchain

static size_t chain_smem(bool prec32) {
  return prec32 ? sizeof(fxchain::Smem<float>) : sizeof(fxchain::Smem<double>);
}

void fx_chain_launch(const fx_dev* devs, const fx_unit* units, int nunits, int max_blocks, bool prec32, cudaStream_t s) {
  const int nblocks = std::max(1, std::min(nunits, max_blocks));
  if (prec32) fxchain::k_chain_batch<float><<<nblocks, fxchain::NTHREADS, chain_smem(true), s>>>(devs, units, nunits);
  else fxchain::k_chain_batch<double><<<nblocks, fxchain::NTHREADS, chain_smem(false), s>>>(devs, units, nunits);
}
void fx_chain_launch_one(const fx_dev& d, int steps, int max_blocks, cudaStream_t s) {
  const int nunits = steps * d.nchem * ((d.nr + fxchain::ROWS - 1) / fxchain::ROWS);
  const int nblocks = std::max(1, std::min(nunits, max_blocks));
  if (d.prec32) fxchain::k_chain_one<float><<<nblocks, fxchain::NTHREADS, chain_smem(true), s>>>(d, steps);
  else fxchain::k_chain_one<double><<<nblocks, fxchain::NTHREADS, chain_smem(false), s>>>(d, steps);
}

// Resident blocks of a kernel, after raising its dynamic shared memory limit.
template <class K>
static int chain_blocks_of(K kernel, size_t smem, int nsm, int* out) {
  int per = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, fxchain::NTHREADS, smem) != cudaSuccess || per < 1)
    return -1;
  *out = per * nsm;
  return 0;
}
// Resident blocks of the kernels of one precision on this device (the fewer
// of the one-domain and the batch form): the units in flight.
int fx_chain_blocks(bool prec32, int* out) {
  int dev = 0, nsm = 0, a = 0, b = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
  const size_t smem = chain_smem(prec32);
  if (prec32 ? (chain_blocks_of(fxchain::k_chain_one<float>, smem, nsm, &a) ||
                chain_blocks_of(fxchain::k_chain_batch<float>, smem, nsm, &b))
             : (chain_blocks_of(fxchain::k_chain_one<double>, smem, nsm, &a) ||
                chain_blocks_of(fxchain::k_chain_batch<double>, smem, nsm, &b)))
    return -1;
  *out = std::min(a, b);
  return 0;
}
