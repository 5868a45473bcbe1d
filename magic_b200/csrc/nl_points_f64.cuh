// FP64 point formulas and reductions shared by the phi-stage kernels
// (nl_bouss.cuh, nl_anel_f64.cu) and the grid-space drop-ins (nonlinear.cu).
#pragma once

#include "common.cuh"

namespace mt {

// ------------------------------------------------------------ point formulas

struct BoussIn {
  double vr, vt, vp, cvr, cvt, cvp, s, br, bt, bp, cbr, cbt, cbp, xi;
};
struct BoussOut {
  double o[12];  // Advr Advt Advp VSr VSt VSp VxBr VxBt VxBp VXir VXit VXip
};

// magic_torch/get_nl.py:57-85
__device__ __forceinline__ void bouss_point(const BoussIn& f, double or2, double or4, double ost2,
                                            double LFfac, bool mag, BoussOut& r) {
  double LFr = 0.0, LFt = 0.0, LFp = 0.0;
  if (mag) {
    LFr = LFfac * ost2 * (f.cbt * f.bp - f.cbp * f.bt);
    LFt = LFfac * or4 * (f.cbp * f.br - f.cbr * f.bp);
    LFp = LFfac * or4 * (f.cbr * f.bt - f.cbt * f.br);
  }
  r.o[0] = -ost2 * (f.cvt * f.vp - f.cvp * f.vt) + LFr;
  r.o[1] = -or4 * (f.cvp * f.vr - f.cvr * f.vp) + LFt;
  r.o[2] = -or4 * (f.cvr * f.vt - f.cvt * f.vr) + LFp;
  r.o[3] = f.vr * f.s;
  r.o[4] = or2 * f.vt * f.s;
  r.o[5] = or2 * f.vp * f.s;
  r.o[6] = ost2 * (f.vt * f.bp - f.vp * f.bt);
  r.o[7] = or4 * (f.vp * f.br - f.vr * f.bp);
  r.o[8] = or4 * (f.vr * f.bt - f.vt * f.br);
  r.o[9] = f.vr * f.xi;
  r.o[10] = or2 * f.vt * f.xi;
  r.o[11] = or2 * f.vp * f.xi;
}

// magic_torch/courant.py:25-77; mode 0 non-magnetic, 1 damped, 2 undamped.
__device__ __forceinline__ void courant_point(int mode, double vr, double vt, double vp, double br,
                                              double bt, double bp, double or2, double or4,
                                              double orho1, double orho2, double ost2,
                                              double LFfac, double cf2, double af2, double valri2,
                                              double valhi2, double& vr2, double& vh2) {
  double vflr2 = orho2 * vr * vr;
  double vflh2 = (vt * vt + vp * vp) * ost2 * orho2;
  if (mode == 0) {
    vr2 = cf2 * or4 * vflr2;
    vh2 = cf2 * or2 * vflh2;
    return;
  }
  double valr = br * br * LFfac * orho1;
  double valh2 = (bt * bt + bp * bp) * LFfac * ost2 * orho1;
  double valr2 = valr, valh2m = valh2;
  if (mode == 1) {
    valr2 = valr * valr / (valr + valri2);
    valh2m = valh2 * valh2 / (valh2 + valhi2);
  }
  vr2 = or4 * (cf2 * vflr2 + af2 * valr2);
  vh2 = or2 * (cf2 * vflh2 + af2 * valh2m);
}

__device__ __forceinline__ double block_max(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < nw ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v;  // valid in thread 0
}

// Block-wide maxima of two values at once (one pass through `red`, >= 2 x 16
// doubles); the results are valid in thread 0.
__device__ __forceinline__ void block_max2(double& a, double& b, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    red[w] = a;
    red[16 + w] = b;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    a = threadIdx.x < nw ? red[threadIdx.x] : 0.0;
    b = threadIdx.x < nw ? red[16 + threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
      b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
  }
}

__device__ __forceinline__ void atomic_max_pos(unsigned long long* a, double v) {
  v = v + 0.0;  // -0 -> +0: bit patterns of non-negative doubles order like integers
  atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

}  // namespace mt
