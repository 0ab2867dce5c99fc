// The order in which a launch of the solute sweep hands out its units (strip
// s of step jj; fx_ade.cu, fx_ade_chain.cu). Plain C++, for the kernels and
// the host.
//
// A unit can start when its west strip of the same step and its own strip of
// the step before are some way along: in the model of fx_ade_start by 37 and 48
// warp steps, so unit (jj, s) at 48 jj + 37 s. Handed out step by step,
// the last strips of a step hold their warps or blocks for thousands of warp
// steps before they can start, while units of later steps that could run are
// not handed out yet (sweep of 4096 x 4096 cells, 20 steps in FP64 1.99 ms a
// step, 63 in FP32 0.65; of 1000 x 700, 24 in FP64 0.190; in the order below
// 1.50, 0.545 and 0.141, all else equal). So units go out by t = jj + floor(3 s / 4), their start
// in units of 48 warp steps, and within a t by step, then strip. Every unit
// that one waits for, (jj, s - 1), (jj - 1, s) and (jj - 1, s + 1), comes
// earlier: t is one less, or the same with a smaller step or strip.
#pragma once

#ifdef __CUDACC__
#define FX_ORDER_FN __host__ __device__ inline
#else
#define FX_ORDER_FN inline
#endif

// How far a caller is: the t it is at and the index of its first unit.
struct fx_unit_walk {
  int t, base;
};

// Unit i (not below an earlier i of the same walk) of steps x strips units.
FX_ORDER_FN void fx_unit_at(int i, int steps, int strips, fx_unit_walk& w, int& jj, int& s) {
  int hi;
  for (;;) {
    // strips with a step 0 <= t - floor(3 s / 4) < steps
    const int past = w.t - steps + 1;
    const int lo = past > 0 ? (4 * past + 2) / 3 : 0;
    hi = (4 * w.t + 3) / 3;
    hi = hi < strips - 1 ? hi : strips - 1;
    const int n = hi - lo + 1;
    if (i < w.base + n) break;
    w.base += n;
    ++w.t;
  }
  s = hi - (i - w.base);  // by step: the last strip first
  // strips 4 a and 4 a + 1 are at the same step: by strip
  if ((s & 3) == 1) --s;
  else if ((s & 3) == 0 && s < hi) ++s;
  jj = w.t - ((3 * s) >> 2);
}
