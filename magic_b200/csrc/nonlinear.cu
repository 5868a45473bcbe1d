// Grid-space nonlinear terms: k_get_nl / k_get_nl_anel / k_courant_grid, the
// formulas of the fused phi stages (magic_torch/get_nl.py:57-87,
// get_nl_anel.py:63-136, courant.py:25-77) on grids held in HBM, for the drop-in
// get_nl / get_nl_anel / courant_check, and the Courant steps of a stage.
#include <algorithm>

#include "fourier.cuh"
#include "nl_points_f64.cuh"

namespace mt {

int launch_nl_bouss(bool mag, bool chem, const NlBoussArgs& a, cudaStream_t st) {
  return a.split_io ? launch_nl_bouss_oz(mag, chem, a, st) : launch_nl_bouss_f64(mag, chem, a, st);
}

__global__ void k_courant_finish(int n_r, const unsigned long long* vr2, const unsigned long long* vh2,
                                 const double* delxr2, const double* delxh2, double* dtr,
                                 double* dth) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_r) return;
  double a = __longlong_as_double((long long)vr2[r]);
  double b = __longlong_as_double((long long)vh2[r]);
  dtr[r] = a > 0.0 ? sqrt(delxr2[r] / a) : 1e10;  // magic_torch/courant.py:122-125
  dth[r] = b > 0.0 ? sqrt(delxh2[r] / b) : 1e10;
}

int launch_courant_finish(int n_r, const unsigned long long* vr2, const unsigned long long* vh2,
                          const double* delxr2, const double* delxh2, double* dtr, double* dth,
                          cudaStream_t st) {
  k_courant_finish<<<(n_r + 127) / 128, 128, 0, st>>>(n_r, vr2, vh2, delxr2, delxh2, dtr, dth);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

// ---------------------------------------------------- grid-space drop-ins


__global__ void k_get_nl(GridNlArgs a) {
  int64_t total = (int64_t)a.n_r * a.nt * a.np;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(i / ((int64_t)a.nt * a.np));
    int th = (int)((i / a.np) % a.nt);
    BoussIn f;
    f.vr = a.in[0][i]; f.vt = a.in[1][i]; f.vp = a.in[2][i];
    f.cvr = a.in[3][i]; f.cvt = a.in[4][i]; f.cvp = a.in[5][i];
    f.s = a.in[6][i];
    f.br = a.in[7][i]; f.bt = a.in[8][i]; f.bp = a.in[9][i];
    f.cbr = a.in[10][i]; f.cbt = a.in[11][i]; f.cbp = a.in[12][i];
    f.xi = a.in[13][i];
    BoussOut o;
    bouss_point(f, a.or2[r], a.or4[r], a.ost2[th], a.LFfac, true, o);
#pragma unroll
    for (int q = 0; q < 12; ++q) a.out[q][i] = o.o[q];
  }
}

// magic_torch/get_nl_anel.py:63-134
__global__ void k_get_nl_anel(GridNlArgs a) {
  int64_t total = (int64_t)a.n_r * a.nt * a.np;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(i / ((int64_t)a.nt * a.np));
    int th = (int)((i / a.np) % a.nt);
    const double vr = a.in[0][i], vt = a.in[1][i], vp = a.in[2][i];
    const double dvrdr = a.in[3][i], dvtdr = a.in[4][i], dvpdr = a.in[5][i];
    const double dvrdt = a.in[6][i], dvrdp = a.in[7][i], dvtdp = a.in[8][i], dvpdp = a.in[9][i];
    const double cvr = a.in[10][i], s = a.in[11][i], xi = a.in[12][i];
    const double br = a.in[13][i], bt = a.in[14][i], bp = a.in[15][i];
    const double cbr = a.in[16][i], cbt = a.in[17][i], cbp = a.in[18][i];
    const double R = a.r[r], or1 = a.or1[r], or2 = a.or2[r], or4 = a.or4[r];
    const double beta = a.beta[r], orho1 = a.orho1[r], otemp1 = a.otemp1[r];
    const double visc = a.visc[r], lam = a.lambda_[r];
    const double ost2 = a.ost2[th], cosn = a.cosn[th], LF = a.LFfac;
    double LFr = LF * ost2 * (cbt * bp - cbp * bt);
    double LFt = LF * or4 * (cbp * br - cbr * bp);
    double LFp = LF * or4 * (cbr * bt - cbt * br);
    double Advr = -or2 * orho1 * (vr * (dvrdr - (2.0 * or1 + beta) * vr) +
                                  ost2 * (vt * (dvrdt - R * vt) + vp * (dvrdp - R * vp)));
    double Advt = or4 * orho1 * (-vr * (dvtdr - beta * vt) + vt * (cosn * vt + dvpdp + dvrdr) +
                                 vp * (cosn * vp - dvtdp));
    double Advp = or4 * orho1 * (-vr * (dvpdr - beta * vp) - vt * (dvtdp + cvr) - vp * dvpdp);
    a.out[0][i] = Advr + LFr;
    a.out[1][i] = Advt + LFt;
    a.out[2][i] = Advp + LFp;
    a.out[3][i] = vr * s;
    a.out[4][i] = or2 * vt * s;
    a.out[5][i] = or2 * vp * s;
    a.out[6][i] = orho1 * ost2 * (vt * bp - vp * bt);
    a.out[7][i] = orho1 * or4 * (vp * br - vr * bp);
    a.out[8][i] = orho1 * or4 * (vr * bt - vt * br);
    a.out[9][i] = vr * xi;
    a.out[10][i] = or2 * vt * xi;
    a.out[11][i] = or2 * vp * xi;
    double prefac = a.ViscHeatFac * or4 * orho1 * otemp1 * visc;
    double beta_r = beta * R;
    double e_rr = dvrdr - (2.0 * or1 + beta) * vr;
    double e_tt = cosn * vt + dvpdp + dvrdr - or1 * vr;
    double e_pp = dvpdp + cosn * vt + or1 * vr;
    double e_tp = 2.0 * dvtdp + cvr - 2.0 * cosn * vp;
    double e_rt = R * dvtdr - (2.0 + beta_r) * vt + or1 * dvrdt;
    double e_rp = R * dvpdr - (2.0 + beta_r) * vp + or1 * dvrdp;
    double bv = beta * vr;
    double heat = prefac * (2.0 * e_rr * e_rr + 2.0 * e_tt * e_tt + 2.0 * e_pp * e_pp +
                            e_tp * e_tp + ost2 * (e_rt * e_rt + e_rp * e_rp) -
                            2.0 * (1.0 / 3.0) * bv * bv);
    if (a.l_mag && a.OhmLossFac != 0.0)
      heat += a.OhmLossFac * lam * or2 * otemp1 * (or2 * cbr * cbr + ost2 * (cbt * cbt + cbp * cbp));
    a.out[12][i] = heat;
  }
}

int launch_get_nl_grid(bool anel, const GridNlArgs& a, cudaStream_t st) {
  int64_t total = (int64_t)a.n_r * a.nt * a.np;
  int blocks = (int)std::min<int64_t>((total + 255) / 256, kSms * 16);
  if (blocks < 1) blocks = 1;
  if (anel) k_get_nl_anel<<<blocks, 256, 0, st>>>(a);
  else k_get_nl<<<blocks, 256, 0, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}


// one CTA per (level, slab of theta rows)
__global__ void k_courant_grid(CourantGridArgs a) {
  __shared__ double red[32];
  const int r = blockIdx.y;
  const int64_t per = (int64_t)a.nt * a.np;
  const int64_t base = (int64_t)r * per;
  const double valri2 = a.valfac / a.delxr2[r], valhi2 = a.valfac / a.delxh2[r];
  double mr = 0.0, mh = 0.0;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < per;
       j += (int64_t)gridDim.x * blockDim.x) {
    int th = (int)(j / a.np);
    int64_t i = base + j;
    double br = 0.0, bt = 0.0, bp = 0.0;
    if (a.mode != 0) { br = a.br[i]; bt = a.bt[i]; bp = a.bp[i]; }
    double vr2, vh2;
    courant_point(a.mode, a.vr[i], a.vt[i], a.vp[i], br, bt, bp, a.or2[r], a.or4[r], a.orho1[r],
                  a.orho2[r], a.ost2[th], a.LFfac, a.cf2, a.af2, valri2, valhi2, vr2, vh2);
    mr = fmax(mr, vr2);
    mh = fmax(mh, vh2);
  }
  double v = block_max(mr, red);
  if (threadIdx.x == 0) atomic_max_pos(&a.vr2max[r], v);
  v = block_max(mh, red);
  if (threadIdx.x == 0) atomic_max_pos(&a.vh2max[r], v);
}

int launch_courant_grid(const CourantGridArgs& a, cudaStream_t st) {
  int64_t per = (int64_t)a.nt * a.np;
  int bx = (int)std::min<int64_t>((per + 255) / 256, 32);
  dim3 grid(bx, a.n_r);
  k_courant_grid<<<grid, 256, 0, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

}  // namespace mt
