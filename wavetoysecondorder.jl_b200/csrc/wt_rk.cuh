// wt_rk.cuh -- the RK4 stage updates of one node, shared by the kernels that fuse them.
#pragma once
#include "wt_common.cuh"

namespace wt {

// Low-storage classic RK4 stage update of node n, with the words it reads passed in
// (yv = y[n], accv = acc[n], compv = comp[n]; only those the stage reads need to be
// valid).  Without compensation acc holds y + partial increments.  With it (comp, FP32
// state) acc holds the increment of the step alone and the final y + increment is a
// Kahan sum; comp holds the low part the FP32 y lost (the state is y + comp), so that
// small increments are not lost to the rounding of y over many steps.  Returns the
// value the stage wrote (the next stage's input, or the new state).
template <typename real>
__device__ __forceinline__ real rk_epilogue_v(int stage, double dt, real k, real yin, real yv, real accv, real compv,
                                              real* y, real* acc, real* out, real* comp, long long n,
                                              unsigned int* nonfinite) {
  real v;
  if (comp) {
    if (stage == 0) {
      v = yin + (real)(0.5 * dt) * k;
      out[n] = v;
      acc[n] = (real)(dt / 6.0) * k;
    } else if (stage == 1) {
      v = yv + (real)(0.5 * dt) * k;
      out[n] = v;
      acc[n] = accv + (real)(dt / 3.0) * k;
    } else if (stage == 2) {
      v = yv + (real)dt * k;
      out[n] = v;
      acc[n] = accv + (real)(dt / 3.0) * k;
    } else {
      const real inc = accv + (real)(dt / 6.0) * k;
      const real t = inc + compv;
      v = yv + t;
      comp[n] = t - (v - yv);
      y[n] = v;
      if (nonfinite && !isfinite((double)v)) atomicOr(nonfinite, 1u);
    }
    return v;
  }
  if (stage == 0) {
    v = yin + (real)(0.5 * dt) * k;
    out[n] = v;
    acc[n] = yin + (real)(dt / 6.0) * k;
  } else if (stage == 1) {
    v = yv + (real)(0.5 * dt) * k;
    out[n] = v;
    acc[n] = accv + (real)(dt / 3.0) * k;
  } else if (stage == 2) {
    v = yv + (real)dt * k;
    out[n] = v;
    acc[n] = accv + (real)(dt / 3.0) * k;
  } else {
    v = accv + (real)(dt / 6.0) * k;
    y[n] = v;
    if (nonfinite && !isfinite((double)v)) atomicOr(nonfinite, 1u);
  }
  return v;
}

// The same of the compensated FP32 form (the Phi side, K1): the state is (y, comp) =
// (high, low part) and the stage the next K1 reads is its high part plus out = low part +
// c dt k; the step's final sum is formed in FP64 and split again.  hi: this node's high
// part of the state (the K1 input); stage 2 copies it into hcopy, which stage 3 reads.
__device__ __forceinline__ void rk_epilogue_cp_v(int stage, double dt, float k, float hi, float lo, float accv,
                                                 float* y, float* acc, float* out, float* comp, float* hcopy,
                                                 long long n, unsigned int* nonfinite) {
  if (stage == 0) {
    out[n] = lo + (float)(0.5 * dt) * k;
    acc[n] = (float)(dt / 6.0) * k;
  } else if (stage == 1) {
    out[n] = lo + (float)(0.5 * dt) * k;
    acc[n] = accv + (float)(dt / 3.0) * k;
  } else if (stage == 2) {
    out[n] = lo + (float)dt * k;
    acc[n] = accv + (float)(dt / 3.0) * k;
    hcopy[n] = hi;
  } else {
    const float inc = accv + (float)(dt / 6.0) * k;
    const double v = (double)hi + ((double)lo + (double)inc);
    const float h = (float)v;
    y[n] = h;
    comp[n] = (float)(v - (double)h);
    if (nonfinite && !isfinite(h)) atomicOr(nonfinite, 1u);
  }
}

}  // namespace wt
