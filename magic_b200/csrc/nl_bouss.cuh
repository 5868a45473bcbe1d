// The fused phi stage of the Boussinesq radial loop in FP64: the Fourier rows
// written by the Legendre synthesis are expanded and inverse-FFT'd in shared
// memory (phi_fft.cuh), the get_nl products (magic_torch/get_nl.py:57-87) and
// the Courant maxima (magic_torch/courant.py:25-77) are formed point by point,
// and the products are forward-FFT'd and truncated to n_m modes for the
// Legendre analysis.  Grids never reach HBM.  Instantiated per row layout in
// nl_bouss_f64.cu (FP64 contractions) and nl_bouss_oz.cu (digit-split ones).
#pragma once

#include "fourier.cuh"
#include "nl_points_f64.cuh"
#include "phi_fft.cuh"

namespace mt {

template <bool MAG, bool CHEM>
struct BoussFields {
  static constexpr int NFI = (MAG ? 6 : 0) + 7 + (CHEM ? 1 : 0);
  static constexpr int NFO = 6 + (MAG ? 3 : 0) + (CHEM ? 3 : 0);
  static constexpr int NB = NFI > NFO ? NFI : NFO;  // rows of the shared buffer
  static constexpr int IV = MAG ? 6 : 0;            // row of vr
};

// One CTA per (theta row, level).  Block-wide phases: load with the real-row
// pre-processing, inverse row FFTs (phi_fft.cuh), products, forward row FFTs,
// store; two CTAs of 256 threads or four of 128 share an SM (where their rows fit
// its shared memory), so one's loads overlap another's arithmetic.
template <bool MAG, bool CHEM, bool SPLIT_IO, class SH, int T>
__global__ void __launch_bounds__(T, 512 / T) k_nl_bouss(NlBoussArgs a) {
  using BF = BoussFields<MAG, CHEM>;
  constexpr int NFI = BF::NFI, NFO = BF::NFO;
  extern __shared__ double smem[];
  __shared__ double red[32];
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem);  // NB rows, S apart
  const Tables& t = a.t;
  const SH sh(t);
  const int H = sh.H, S = sh.S, M = t.n_m;
  cplx<double>* tw1 = buf + BF::NB * S;
  cplx<double>* twN = tw1 + (sh.A - 1) * sh.Ns;
  // levels run fastest through the grid: the CTAs resident at one time read
  // (and write) whole runs of levels of a few theta rows, contiguous in HBM
  const int row = blockIdx.y, r = blockIdx.x, tid = threadIdx.x;
  phi_twiddles_to_smem(tw1, sh, t);
  // k = 0 coefficients of Fourier row `row`, level r, and the doubles from one k
  // to the next
  auto at = [&](int row, int r) -> const double* {
    if constexpr (SPLIT_IO)  // [m][north|south][theta pair][level, field]
      return a.Fs + (int64_t)(row & 1) * a.fs_c + (int64_t)(row >> 1) * a.fs_j +
             (int64_t)r * 2 * NFI;
    else
      return reinterpret_cast<const double*>(a.F + (int64_t)row * a.f_row + (int64_t)r * NFI);
  };
  const int64_t pitch = SPLIT_IO ? a.fs_m : 2 * a.f_m;
  phi_prefetch<NFI, T>(M, pitch, at);
  const double* x0 = at(row, r);
  auto ldF = [&](int k, int f) {
    const double2 x = __ldg(reinterpret_cast<const double2*>(x0 + (int64_t)k * pitch) + f);
    return cplx<double>{x.x, x.y};
  };
  phi_load_rows<NFI, T>(buf, sh, M, twN, ldF);
  phi_inverse(buf, NFI, sh, tw1);

  const double or2 = a.or2[r], or4 = a.or4[r], ost2 = t.ost2[row];
  const double orho1 = a.orho1[r], orho2 = a.orho2[r];
  const double valri2 = a.valfac / a.delxr2[r], valhi2 = a.valfac / a.delxh2[r];
  const double LF = a.LFfac_r ? a.LFfac_r[r] : a.LFfac;
  double mr = 0.0, mh = 0.0;
  auto point = [&](const double (&v)[NFI], double (&out)[NFO]) {
    BoussIn fi;
    constexpr int iv = BF::IV;
    if constexpr (MAG) {
      fi.br = v[0]; fi.bt = v[1]; fi.bp = v[2]; fi.cbr = v[3]; fi.cbt = v[4]; fi.cbp = v[5];
    } else {
      fi.br = fi.bt = fi.bp = fi.cbr = fi.cbt = fi.cbp = 0.0;
    }
    fi.vr = v[iv]; fi.vt = v[iv + 1]; fi.vp = v[iv + 2];
    fi.cvr = v[iv + 3]; fi.cvt = v[iv + 4]; fi.cvp = v[iv + 5];
    fi.s = v[iv + 6];
    fi.xi = 0.0;
    if constexpr (CHEM) fi.xi = v[iv + 7];
    double vr2, vh2;
    courant_point(a.cour_mode, fi.vr, fi.vt, fi.vp, fi.br, fi.bt, fi.bp, or2, or4, orho1, orho2,
                  ost2, LF, a.cf2, a.af2, valri2, valhi2, vr2, vh2);
    mr = fmax(mr, vr2);
    mh = fmax(mh, vh2);
    BoussOut o;
    bouss_point(fi, or2, or4, ost2, LF, MAG, o);
#pragma unroll
    for (int q = 0; q < 6; ++q) out[q] = o.o[q];
    if constexpr (MAG) { out[6] = o.o[6]; out[7] = o.o[7]; out[8] = o.o[8]; }
    if constexpr (CHEM) {
      constexpr int c = MAG ? 9 : 6;
      out[c] = o.o[9]; out[c + 1] = o.o[10]; out[c + 2] = o.o[11];
    }
  };
  phi_points<NFI, NFO, T>(buf, sh, point);
  block_max2(mr, mh, red);
  if (tid == 0) {
    atomic_max_pos(&a.vr2max[r], mr);
    atomic_max_pos(&a.vh2max[r], mh);
  }
  if (r == 0 || r == a.n_r - 1) return;  // boundary levels: Courant only
  __syncthreads();
  phi_forward(buf, NFO, sh, tw1);
  // radial components (Advr, VSr, VxBr, VXir) are scalar analyses
  const double ws = t.wq[row] / (2 * H), wv = t.wq_v[row] / (2 * H);
  double2* Gr = SPLIT_IO
                    ? reinterpret_cast<double2*>(a.Gs + (int64_t)(row & 1) * a.g_h +
                                                 (int64_t)(row >> 1) * a.g_j +
                                                 (int64_t)(r - 1) * a.g_level)
                    : a.G + (int64_t)row * a.g_row + (int64_t)(r - 1) * NFO;
  const int64_t gm = SPLIT_IO ? a.g_m2 / 2 : a.g_m;  // double2 stride between orders
  phi_store_rows<NFO, T>(buf, sh, M, twN, [&](int k, int o, cplx<double> X) {
    const bool radial = (o == 0 || o == 3 || (MAG && o == 6) || (CHEM && o == (MAG ? 9 : 6)));
    const double w = radial ? ws : wv;
    Gr[k * gm + o] = make_double2(w * X.x, w * X.y);
  });
}

template <bool MAG, bool CHEM, bool SPLIT_IO, class SH, int T>
static int launch_nl_bouss_s(const NlBoussArgs& a, cudaStream_t st) {
  const size_t sm = ((size_t)BoussFields<MAG, CHEM>::NB * phi_row_len(a.t) + phi_tw_len(a.t)) *
                    sizeof(double2);
  auto kern = k_nl_bouss<MAG, CHEM, SPLIT_IO, SH, T>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
  dim3 grid(a.n_r, a.t.n_theta);
  kern<<<grid, T, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <bool MAG, bool CHEM, bool SPLIT_IO>
static int launch_nl_bouss_t(const NlBoussArgs& a, cudaStream_t st) {
  if (phi_shape_static(a.t)) switch (a.t.fft_b) {
#define X(b) \
  case b: return launch_nl_bouss_s<MAG, CHEM, SPLIT_IO, PhiShape<16, b, 2>, 256>(a, st);
      MT_PHI_STATIC_B(X)
#undef X
      default: break;
    }
  const int r = phi_max_radix(a.t);
  if (r <= 12) return launch_nl_bouss_s<MAG, CHEM, SPLIT_IO, PhiShapeRt<12>, 128>(a, st);
  if (r <= 18) return launch_nl_bouss_s<MAG, CHEM, SPLIT_IO, PhiShapeRt<18>, 256>(a, st);
  return launch_nl_bouss_s<MAG, CHEM, SPLIT_IO, PhiShapeRt<27>, 256>(a, st);
}

template <bool SPLIT_IO>
static int launch_nl_bouss_io(bool mag, bool chem, const NlBoussArgs& a, cudaStream_t st) {
  if (mag)
    return chem ? launch_nl_bouss_t<true, true, SPLIT_IO>(a, st)
                : launch_nl_bouss_t<true, false, SPLIT_IO>(a, st);
  return chem ? launch_nl_bouss_t<false, true, SPLIT_IO>(a, st)
              : launch_nl_bouss_t<false, false, SPLIT_IO>(a, st);
}

}  // namespace mt
