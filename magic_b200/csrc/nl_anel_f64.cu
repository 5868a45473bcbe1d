// The FP64 phi stage of the anelastic radial loop, on the rows of the FP64 and of the
// digit-split contractions.
#include <algorithm>

#include "nl_point.cuh"
#include "nl_points_f64.cuh"
#include "phi_fft.cuh"
#include "split_kernels.cuh"

namespace mt {

// One CTA (256 threads) per (theta row, level): the synthesis wrote this
// hemisphere's Fourier rows of the grid fields in FP64 (NlAnelArgs::Fs64; field
// order of nl_point.cuh), the kernel inverse-transforms them in place
// (phi_fft.cuh), evaluates get_nl_anel (magic_torch/get_nl_anel.py:63-136, viscous
// and Ohmic heating included) and the Courant maxima (magic_torch/courant.py:25-77)
// at every grid point in FP64, and forward-transforms the 7 to 13 products into
// the weighted rows the analysis reads (NlAnelArgs::G64).  Shared memory holds
// only the rows (the twiddle tables are read through L1), so that two CTAs
// share an SM without magnetic field at n_phi = 1152.  Velocity, its
// derivatives and cvr are zero on the two boundary levels (radial_loop_anel
// synthesises them on the bulk levels only, magic_torch/step_time.py:
// 1233-1316); the phi-derivative fields get their 1/sin^2(theta) factor here
// (torpol_to_dphspat, magic_torch/sht.py:725-743).
constexpr int kNlAnelThreads = 256;

template <bool MAG, bool CHEM, class SH>
__global__ void __launch_bounds__(kNlAnelThreads, 2) k_nl_anel_f64(NlAnelArgs a) {
  using F = AnelFields<MAG, CHEM>;
  constexpr int NFI = F::NFI, NFO = F::NFO, T = kNlAnelThreads;
  extern __shared__ double smem[];
  __shared__ double red[32];
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem);
  const Tables& t = a.t;
  const SH sh(t);
  const int N = t.n_phi, M = t.n_m;
  const cplx<double>* tw1 = reinterpret_cast<const cplx<double>*>(t.phi_tw1);
  const cplx<double>* twN = reinterpret_cast<const cplx<double>*>(t.twiddle);
  const int r = blockIdx.x, row = blockIdx.y, tid = threadIdx.x;
  auto at = [&](int row, int r) {
    return a.Fs64 + (int64_t)(row & 1) * a.fs_c + (int64_t)(row >> 1) * a.fs_j +
           (int64_t)r * 2 * NFI;
  };
  phi_prefetch<NFI, T>(M, a.fs_m, at);
  const double* frow = at(row, r);
  phi_load_rows<NFI, T>(buf, sh, M, twN, [&](int k, int f) {
    const double2 x = __ldg(reinterpret_cast<const double2*>(frow + (int64_t)k * a.fs_m) + f);
    return cplx<double>{x.x, x.y};
  });
  phi_inverse(buf, NFI, sh, tw1);

  const bool bnd = r == 0 || r == a.n_r - 1;
  AnelLevel<double> L;
  L.R = a.r[r];
  L.or1 = a.or1[r];
  L.or2 = a.or2[r];
  L.or4 = a.or4[r];
  L.beta = a.beta[r];
  L.orho1 = a.orho1[r];
  L.otemp1 = a.otemp1[r];
  L.visc = a.visc[r];
  L.lam = a.lambda_[r];
  L.LF = a.LFfac;
  L.vhf = a.ViscHeatFac;
  L.ohm = a.OhmLossFac;
  const double ost2 = t.ost2[row], cosn = t.cosn[row], orho2 = a.orho2[r];
  const double valri2 = a.valfac / a.delxr2[r], valhi2 = a.valfac / a.delxh2[r];
  double mr = 0.0, mh = 0.0;
  auto point = [&](double (&v)[NFI], double (&o)[NFO]) {
    if (bnd) {
#pragma unroll
      for (int f = 0; f <= 10; ++f) v[f] = 0.0;  // velocity, derivatives, cvr
    }
    v[8] *= ost2;  // dvtdp, dvpdp: torpol_to_dphspat's 1/sin^2
    v[9] *= ost2;
    double vr2, vh2;
    if constexpr (MAG)
      courant_point(a.cour_mode, v[0], v[1], v[2], v[F::IB], v[F::IB + 1], v[F::IB + 2], L.or2,
                    L.or4, L.orho1, orho2, ost2, L.LF, a.cf2, a.af2, valri2, valhi2, vr2, vh2);
    else
      courant_point(0, v[0], v[1], v[2], 0.0, 0.0, 0.0, L.or2, L.or4, L.orho1, orho2, ost2, L.LF,
                    a.cf2, a.af2, valri2, valhi2, vr2, vh2);
    mr = fmax(mr, vr2);
    mh = fmax(mh, vh2);
    anel_point<double, MAG, CHEM>(v, L, ost2, cosn, o);
  };
  phi_points<NFI, NFO, T>(buf, sh, point);
  block_max2(mr, mh, red);
  if (tid == 0) {
    atomic_max_pos(&a.vr2max[r], mr);
    atomic_max_pos(&a.vh2max[r], mh);
  }
  if (bnd) return;  // boundary levels: Courant only
  __syncthreads();
  phi_forward(buf, NFO, sh, tw1);
  const double ws = t.wq[row] / N, wv = t.wq_v[row] / N;
  double* Gr = a.G64 + (int64_t)(row & 1) * a.g_h + (int64_t)(row >> 1) * a.g_j +
               (int64_t)(r - 1) * a.g_level;
  phi_store_rows<NFO, T>(buf, sh, M, twN, [&](int k, int o, cplx<double> X) {
    const double w = F::radial(o) ? ws : wv;
    reinterpret_cast<double2*>(Gr + k * a.g_m)[o] = make_double2(w * X.x, w * X.y);
  });
}

// Dynamic shared memory: the rows (0 if they do not fit, which no n_phi within
// the plan's limit reaches).
size_t nl_anel_f64_smem(const Tables& t, bool mag, bool chem) {
  const int nfi = 12 + (chem ? 1 : 0) + (mag ? 6 : 0), nfo = 7 + (mag ? 3 : 0) + (chem ? 3 : 0);
  const size_t sm = (size_t)std::max(nfi, nfo) * phi_row_len(t) * sizeof(double2);
  return sm <= 227 * 1024 - 32 * sizeof(double) ? sm : 0;
}

template <bool MAG, bool CHEM, class SH>
static int launch_nl_anel_f64_s(const NlAnelArgs& a, cudaStream_t st) {
  const size_t sm = nl_anel_f64_smem(a.t, MAG, CHEM);
  MT_REQUIRE(sm > 0, MT_ERR_UNSUPPORTED, "n_phi too large for the FP64 anelastic phi stage");
  auto kern = k_nl_anel_f64<MAG, CHEM, SH>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
  dim3 grid(a.n_r, a.t.n_theta);
  kern<<<grid, kNlAnelThreads, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <bool MAG, bool CHEM>
static int launch_nl_anel_f64_t(const NlAnelArgs& a, cudaStream_t st) {
  if (phi_shape_static(a.t)) switch (a.t.fft_b) {
#define X(b) case b: return launch_nl_anel_f64_s<MAG, CHEM, PhiShape<16, b, 2>>(a, st);
      MT_PHI_STATIC_B(X)
#undef X
      default: break;
    }
  const int r = phi_max_radix(a.t);
  if (r <= 12) return launch_nl_anel_f64_s<MAG, CHEM, PhiShapeRt<12>>(a, st);
  return r <= 18 ? launch_nl_anel_f64_s<MAG, CHEM, PhiShapeRt<18>>(a, st)
                 : launch_nl_anel_f64_s<MAG, CHEM, PhiShapeRt<27>>(a, st);
}

int launch_nl_anel_f64(bool mag, bool chem, const NlAnelArgs& a, cudaStream_t st) {
  if (mag)
    return chem ? launch_nl_anel_f64_t<true, true>(a, st)
                : launch_nl_anel_f64_t<true, false>(a, st);
  return chem ? launch_nl_anel_f64_t<false, true>(a, st)
              : launch_nl_anel_f64_t<false, false>(a, st);
}

}  // namespace mt
