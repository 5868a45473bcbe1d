// Fused phi stage of the split-precision anelastic radial loop (FP32).
//
// One CTA per (theta row, level), as k_nl_bouss_split_hw: the synthesis
// delivers equatorially symmetric/antisymmetric Fourier rows of the 18 (19
// with composition) grid fields, this kernel forms the hemisphere's rows,
// transforms them (half-warp FFT for n_phi = 256, 384, 512, 768, two-step row FFTs
// otherwise), evaluates get_nl_anel (magic_torch/get_nl_anel.py:41-136,
// viscous and Ohmic heating included) and the Courant maxima at every grid
// point, and writes the weighted Fourier rows of the 10-13 products for the
// analysis.  Velocity, its derivatives and cvr are zero on the two boundary
// levels (radial_loop_anel synthesises them on the bulk levels only); the
// phi-derivative fields get their 1/sin^2(theta) factor here
// (torpol_to_dphspat, magic_torch/sht.py:725-743).
//
// Grid fields (rows 2 f, 2 f + 1 of the synthesis): 0 vr, 1 vt, 2 vp,
// 3 dvrdr, 4 dvtdr, 5 dvpdr, 6 dvrdt, 7 dvrdp, 8 dvtdp, 9 dvpdp, 10 cvr,
// 11 s, [12 xi], then br bt bp cbr cbt cbp.  Products: 0 Advr, 1 Advt,
// 2 Advp, 3 VSr, 4 VSt, 5 VSp, [VxBr VxBt VxBp], [VXir VXit VXip], heat.
#include "fft.cuh"
#include "fft_hw.cuh"
#include "nl_point.cuh"
#include "phi_fft.cuh"
#include "split_kernels.cuh"

namespace mt {

// Constants of one (theta row, level).
struct AnelSplitRow {
  bool bnd;
  AnelLevel<float> L;
  float ost2, cosn, orho2, valri2, valhi2, cf2, af2;
};
__device__ __forceinline__ AnelSplitRow anel_split_row(const NlAnelArgs& a, int row, int r) {
  AnelSplitRow R;
  R.bnd = r == 0 || r == a.n_r - 1;
  AnelLevel<float>& L = R.L;
  L.R = (float)a.r[r];
  L.or1 = (float)a.or1[r];
  L.or2 = (float)a.or2[r];
  L.or4 = (float)a.or4[r];
  L.beta = (float)a.beta[r];
  L.orho1 = (float)a.orho1[r];
  L.otemp1 = (float)a.otemp1[r];
  L.visc = (float)a.visc[r];
  L.lam = (float)a.lambda_[r];
  L.LF = (float)a.LFfac;
  L.vhf = (float)a.ViscHeatFac;
  L.ohm = (float)a.OhmLossFac;
  R.ost2 = (float)a.t.ost2[row];
  R.cosn = (float)a.t.cosn[row];
  R.orho2 = (float)a.orho2[r];
  R.valri2 = (float)(a.valfac / a.delxr2[r]);
  R.valhi2 = (float)(a.valfac / a.delxh2[r]);
  R.cf2 = (float)a.cf2;
  R.af2 = (float)a.af2;
  return R;
}

// One grid point: the fields v (modified: boundary zeros, 1/sin^2), products o,
// Courant terms into mr, mh.
template <bool MAG, bool CHEM>
__device__ __forceinline__ void anel_split_point(const NlAnelArgs& a, const AnelSplitRow& R,
                                                 float* v, float* o, float& mr, float& mh) {
  using F = AnelFields<MAG, CHEM>;
  const AnelLevel<float>& L = R.L;
  if (R.bnd) {
#pragma unroll
    for (int f = 0; f <= 10; ++f) v[f] = 0.f;  // velocity, derivatives, cvr
  }
  v[8] *= R.ost2;  // dvtdp, dvpdp: torpol_to_dphspat's 1/sin^2
  v[9] *= R.ost2;
  float vr2, vh2;
  if constexpr (MAG)
    courant_point_s(a.cour_mode, v[0], v[1], v[2], v[F::IB], v[F::IB + 1], v[F::IB + 2], L.or2,
                    L.or4, L.orho1, R.orho2, R.ost2, L.LF, R.cf2, R.af2, R.valri2, R.valhi2, vr2,
                    vh2);
  else
    courant_point_s(0, v[0], v[1], v[2], 0.f, 0.f, 0.f, L.or2, L.or4, L.orho1, R.orho2, R.ost2,
                    L.LF, R.cf2, R.af2, R.valri2, R.valhi2, vr2, vh2);
  mr = fmaxf(mr, vr2);
  mh = fmaxf(mh, vh2);
  anel_point<float, MAG, CHEM>(v, L, R.ost2, R.cosn, o);
}

// n_phi = 32 Q: half-warp FFTs (fft_hw.cuh).
template <bool MAG, bool CHEM, int Q>
__global__ void __launch_bounds__(AnelFields<MAG, CHEM>::THW) k_nl_anel_split_hw(NlAnelArgs a) {
  using F = AnelFields<MAG, CHEM>;
  constexpr int NFI = F::NFI, NFO = F::NFO, NB = F::NB, T = F::THW;
  extern __shared__ __align__(16) float smemf[];
  __shared__ double red[32];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const int N = t.n_phi, H = N / 2, M = t.n_m, S = H + 1;
  const int row = blockIdx.x, r = blockIdx.y, j = row >> 1;
  const float hs = (row & 1) ? -1.f : 1.f;  // north = sym + asym, south = sym - asym
  const int tid = threadIdx.x;
  cplx<float>* tw2 = buf + NB * S;
  cplx<float>* tw3 = tw2 + 3 * Q;
  cplx<float>* twN = tw3 + 12 * Q;
  hw_twiddles_to_smem<Q>(tw2, tw3, twN, t.twiddle, tid, T);
  const float* fsym = a.Fs + (int64_t)j * a.fs_j + (int64_t)r * 2 * NFI;
#pragma unroll 4
  for (int e = tid; e < NFI * M; e += T) {
    const int k = e / NFI, f = e - k * NFI;
    const float2 sy = __ldg(reinterpret_cast<const float2*>(fsym + k * a.fs_m) + f);
    const float2 as = __ldg(reinterpret_cast<const float2*>(fsym + k * a.fs_m + a.fs_c) + f);
    buf[f * S + hw_swz<Q>(k)] = {sy.x + hs * as.x, sy.y + hs * as.y};
  }
  for (int e = tid; e < NFI * (H - M); e += T) {
    const int k = M + e / NFI, f = e % NFI;
    buf[f * S + hw_swz<Q>(k)] = {0.f, 0.f};
  }
  __syncthreads();
  const int hw = tid >> 4, lane = tid & 15;
  const unsigned mask = 0xFFFFu << (16 * (hw & 1));
  if (hw < NFI) hw_row_fft<Q, true, true>(buf + hw * S, lane, mask, tw2, tw3, twN);
  __syncthreads();
  const AnelSplitRow R = anel_split_row(a, row, r);
  float mr = 0.f, mh = 0.f;
  for (int i = tid; i < H; i += T) {
    const int si = hw_swz<Q>(i);
    cplx<float> zin[NFI];
#pragma unroll
    for (int f = 0; f < NFI; ++f) zin[f] = buf[f * S + si];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v[NFI], o[NFO];
#pragma unroll
      for (int f = 0; f < NFI; ++f) v[f] = h ? zin[f].y : zin[f].x;
      anel_split_point<MAG, CHEM>(a, R, v, o, mr, mh);
      if (!R.bnd) {
#pragma unroll
        for (int q = 0; q < NFO; ++q) {
          if (h) buf[q * S + si].y = o[q];
          else buf[q * S + si].x = o[q];
        }
      }
    }
  }
  double vmr = block_max_d((double)mr, red);
  if (tid == 0) atomicMax(&a.vr2max[r], (unsigned long long)__double_as_longlong(vmr + 0.0));
  double vmh = block_max_d((double)mh, red);
  if (tid == 0) atomicMax(&a.vh2max[r], (unsigned long long)__double_as_longlong(vmh + 0.0));
  if (R.bnd) return;
  __syncthreads();
  if (hw < NFO) hw_row_fft<Q, false, false>(buf + hw * S, lane, mask, tw2, tw3, twN);
  __syncthreads();
  const float ws = (float)(t.wq[row] / N), wv = (float)(t.wq_v[row] / N);
  float* Gr = a.G + (int64_t)(row & 1) * a.g_h + (int64_t)j * a.g_j + (int64_t)(r - 1) * a.g_level;
  for (int e = tid; e < M * NFO; e += T) {
    const int k = e / NFO, o = e - k * NFO;
    const cplx<float>* z = buf + o * S;
    const cplx<float> X = r2c_post(z[hw_swz<Q>(k)], z[hw_swz<Q>((H - k) % H)], twN[k]);
    const float w = F::radial(o) ? ws : wv;
    reinterpret_cast<float2*>(Gr + k * a.g_m)[o] = make_float2(w * X.x, w * X.y);
  }
}

// Any other n_phi (1152 at l_max 383): block-wide row FFTs (phi_fft.cuh).
template <bool MAG, bool CHEM, class SH, int T>
__global__ void __launch_bounds__(T, SH::kMax <= 12 ? 768 / T : 512 / T)
    k_nl_anel_split(NlAnelArgs a) {
  using F = AnelFields<MAG, CHEM>;
  constexpr int NFI = F::NFI, NFO = F::NFO;
  extern __shared__ __align__(16) float smemf[];
  __shared__ double red[32];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const SH sh(t);
  const int N = t.n_phi, M = t.n_m;
  cplx<float>* tw1 = buf + F::NB * sh.S;
  cplx<float>* twN = tw1 + (sh.A - 1) * sh.Ns;
  const int row = blockIdx.x, r = blockIdx.y, j = row >> 1, tid = threadIdx.x;
  const float hs = (row & 1) ? -1.f : 1.f;  // north = sym + asym, south = sym - asym
  phi_twiddles_to_smem(tw1, sh, t);
  const float* fsym = a.Fs + (int64_t)j * a.fs_j + (int64_t)r * 2 * NFI;
  phi_load_rows<NFI, T>(buf, sh, M, twN, [&](int k, int f) {
    const float2 sy = __ldg(reinterpret_cast<const float2*>(fsym + k * a.fs_m) + f);
    const float2 as = __ldg(reinterpret_cast<const float2*>(fsym + k * a.fs_m + a.fs_c) + f);
    return cplx<float>{sy.x + hs * as.x, sy.y + hs * as.y};
  });
  phi_inverse(buf, NFI, sh, tw1);
  const AnelSplitRow R = anel_split_row(a, row, r);
  float mr = 0.f, mh = 0.f;
  auto point = [&](float (&v)[NFI], float (&o)[NFO]) {
    anel_split_point<MAG, CHEM>(a, R, v, o, mr, mh);
  };
  phi_points<NFI, NFO, T>(buf, sh, point);
  double vmr = block_max_d((double)mr, red);
  if (tid == 0) atomicMax(&a.vr2max[r], (unsigned long long)__double_as_longlong(vmr + 0.0));
  double vmh = block_max_d((double)mh, red);
  if (tid == 0) atomicMax(&a.vh2max[r], (unsigned long long)__double_as_longlong(vmh + 0.0));
  if (R.bnd) return;
  __syncthreads();
  phi_forward(buf, NFO, sh, tw1);
  const float ws = (float)(t.wq[row] / N), wv = (float)(t.wq_v[row] / N);
  float* Gr = a.G + (int64_t)(row & 1) * a.g_h + (int64_t)j * a.g_j + (int64_t)(r - 1) * a.g_level;
  phi_store_rows<NFO, T>(buf, sh, M, twN, [&](int k, int o, cplx<float> X) {
    const float w = F::radial(o) ? ws : wv;
    reinterpret_cast<float2*>(Gr + k * a.g_m)[o] = make_float2(w * X.x, w * X.y);
  });
}

template <bool MAG, bool CHEM, int Q>
static int launch_anel_hw(const NlAnelArgs& a, cudaStream_t st) {
  using F = AnelFields<MAG, CHEM>;
  const int H = a.t.n_phi / 2;
  const size_t sm = ((size_t)F::NB * (H + 1) + 15 * Q + H) * sizeof(cplx<float>);
  auto kern = k_nl_anel_split_hw<MAG, CHEM, Q>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
  dim3 grid(a.t.n_theta, a.n_r);
  kern<<<grid, F::THW, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <bool MAG, bool CHEM, class SH, int T>
static int launch_anel_phi(const NlAnelArgs& a, cudaStream_t st) {
  const size_t sm = ((size_t)AnelFields<MAG, CHEM>::NB * phi_row_len(a.t) + phi_tw_len(a.t)) *
                    sizeof(cplx<float>);
  auto kern = k_nl_anel_split<MAG, CHEM, SH, T>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
  dim3 grid(a.t.n_theta, a.n_r);
  kern<<<grid, T, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <bool MAG, bool CHEM>
static int launch_anel_t(const NlAnelArgs& a, cudaStream_t st) {
  switch (a.t.n_phi) {
    case 256: return launch_anel_hw<MAG, CHEM, 8>(a, st);
    case 384: return launch_anel_hw<MAG, CHEM, 12>(a, st);
    case 512: return launch_anel_hw<MAG, CHEM, 16>(a, st);
    case 768: return launch_anel_hw<MAG, CHEM, 24>(a, st);
    default: break;
  }
  return phi_max_radix(a.t) <= 12 ? launch_anel_phi<MAG, CHEM, PhiShapeRt<12>, 128>(a, st)
                                  : launch_anel_phi<MAG, CHEM, PhiShapeRt<27>, 256>(a, st);
}

int launch_nl_anel_split(bool mag, bool chem, const NlAnelArgs& a, cudaStream_t st) {
  if (mag) return chem ? launch_anel_t<true, true>(a, st) : launch_anel_t<true, false>(a, st);
  return chem ? launch_anel_t<false, true>(a, st) : launch_anel_t<false, false>(a, st);
}

}  // namespace mt
