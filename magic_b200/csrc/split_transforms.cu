// phi stage of the split-precision drop-in transforms (FP32).
//
// Rows are (column b, field f) pairs, row r = b * nf + f, matching the row
// order of the split Legendre kernels (row program q = 2 f + re/im of column
// b).  Synthesis: the Legendre GEMM leaves equatorially symmetric and
// antisymmetric Fourier rows (FP32); this kernel forms north = sym + asym or
// south = sym - asym, runs irfft(norm="forward") and writes the FP64 grid
// row.  Analysis: rfft(norm="forward") of the FP64 grid row in FP32, scaled
// by 1/N and by the row's quadrature weight (2 pi w, or 2 pi w / sin^2 for
// vector components), written as north/south Fourier rows for the analysis
// packing kernel.  One CTA = (theta row, up to kPhiRows rows); the FFT is the
// half-warp one (fft_hw.cuh) for n_phi = 256, 384, 512, 768, Stockham passes
// (fft.cuh) where the two steps would be too few transforms of 25 or 27 points
// (launch_split_phi), and the two-step one (phi_fft.cuh) otherwise.
#include "fft_hw.cuh"
#include "phi_fft.cuh"
#include "split_kernels.cuh"

namespace mt {

constexpr int kPhiRows = 14;
constexpr int kPhiThreads = kPhiRows * 16;

template <int Q>
__global__ void __launch_bounds__(kPhiThreads) k_split_to_grid_hw(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const int N = t.n_phi, H = N / 2, M = t.n_m, nt = t.n_theta;
  const int S = H + 1;
  const int row = blockIdx.x, j = row >> 1;
  const float hs = (row & 1) ? -1.f : 1.f;  // north = sym + asym, south = sym - asym
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  const int tid = threadIdx.x;
  cplx<float>* tw2 = buf + kPhiRows * S;
  cplx<float>* tw3 = tw2 + 3 * Q;
  cplx<float>* twN = tw3 + 12 * Q;
  hw_twiddles_to_smem<Q>(tw2, tw3, twN, t.twiddle, tid, kPhiThreads);
  // rows r0 .. r0 + nrow of wavenumber k are contiguous in the synthesis output
  const float* fs = a.Fs + (int64_t)j * a.fs_j + 2 * r0;
  const float rcp = 1.0f / (float)nrow;
  for (int e = tid; e < nrow * M; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    const float2 sy = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m) + q);
    const float2 as = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m + a.fs_c) + q);
    buf[q * S + hw_swz<Q>(k)] = {sy.x + hs * as.x, sy.y + hs * as.y};
  }
  for (int e = tid; e < nrow * (H - M); e += kPhiThreads) {
    const int q = e / (H - M), k = M + e % (H - M);
    buf[q * S + hw_swz<Q>(k)] = {0.f, 0.f};
  }
  __syncthreads();
  const int hw = tid >> 4, lane = tid & 15;
  if (hw < nrow)
    hw_row_fft<Q, true, true>(buf + hw * S, lane, 0xFFFFu << (16 * (hw & 1)), tw2, tw3, twN);
  __syncthreads();
  // one warp per row: z[n] carries grid values 2n, 2n+1 (one 16-byte store)
  const int warp = tid >> 5, l32 = tid & 31;
  for (int q = warp; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    double2* dst = reinterpret_cast<double2*>(a.out[f] + ((int64_t)b * nt + row) * N);
    for (int n = l32; n < H; n += 32) {
      const cplx<float> z = buf[q * S + hw_swz<Q>(n)];
      dst[n] = make_double2((double)z.x, (double)z.y);
    }
  }
}

template <int Q>
__global__ void __launch_bounds__(kPhiThreads) k_split_to_fourier_hw(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const int N = t.n_phi, H = N / 2, M = t.n_m, nt = t.n_theta;
  const int S = H + 1;
  const int row = blockIdx.x, j = row >> 1;
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  const int tid = threadIdx.x;
  cplx<float>* tw2 = buf + kPhiRows * S;
  cplx<float>* tw3 = tw2 + 3 * Q;
  cplx<float>* twN = tw3 + 12 * Q;
  hw_twiddles_to_smem<Q>(tw2, tw3, twN, t.twiddle, tid, kPhiThreads);
  const int warp = tid >> 5, l32 = tid & 31;
  for (int q = warp; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const double2* src = reinterpret_cast<const double2*>(a.in[f] + ((int64_t)b * nt + row) * N);
    for (int n = l32; n < H; n += 32) {
      const double2 v = __ldg(src + n);
      buf[q * S + hw_swz<Q>(n)] = {(float)v.x, (float)v.y};
    }
  }
  __syncthreads();
  const int hw = tid >> 4, lane = tid & 15;
  if (hw < nrow)
    hw_row_fft<Q, false, false>(buf + hw * S, lane, 0xFFFFu << (16 * (hw & 1)), tw2, tw3, twN);
  __syncthreads();
  const float ws = (float)(t.wq[row] / N), wv = (float)(t.wq_v[row] / N);
  float* G = a.G + (int64_t)(row & 1) * a.g_h + (int64_t)j * a.g_j;
  const float rcp = 1.0f / (float)nrow;
  for (int e = tid; e < M * nrow; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const cplx<float>* z = buf + q * S;
    const cplx<float> X = r2c_post(z[hw_swz<Q>(k)], z[hw_swz<Q>((H - k) % H)], twN[k]);
    const float w = (a.vector_mask >> f) & 1 ? wv : ws;
    reinterpret_cast<float2*>(G + k * a.g_m + (int64_t)b * a.g_level)[f] =
        make_float2(w * X.x, w * X.y);
  }
}

// Any other n_phi: block-wide row FFTs (phi_fft.cuh).
template <class SH>
__global__ void __launch_bounds__(kPhiThreads, SH::kMax <= 12 ? 4 : 3)
    k_split_to_grid(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const SH sh(t);
  const int H = sh.H, N = 2 * H, M = t.n_m, nt = t.n_theta, tid = threadIdx.x;
  const int row = blockIdx.x, j = row >> 1;
  const float hs = (row & 1) ? -1.f : 1.f;  // north = sym + asym, south = sym - asym
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  cplx<float>* tw1 = buf + kPhiRows * sh.S;
  cplx<float>* twN = tw1 + (sh.A - 1) * sh.Ns;
  phi_twiddles_to_smem(tw1, sh, t);
  __syncthreads();
  // rows r0 .. r0 + nrow of wavenumber k are contiguous in the synthesis output
  const float* fs = a.Fs + (int64_t)j * a.fs_j + 2 * r0;
  const float rcp = 1.0f / (float)nrow;
  auto ld = [&](int k, int q) {
    const float2 sy = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m) + q);
    const float2 as = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m + a.fs_c) + q);
    return cplx<float>{sy.x + hs * as.x, sy.y + hs * as.y};
  };
#pragma unroll 4
  for (int e = tid; e < (H / 2 + 1) * nrow; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    cplx<float> Xk = {0.f, 0.f}, Xc = {0.f, 0.f};
    if (k < M) Xk = ld(k, q);
    if (k > 0 && H - k < M) Xc = ld(H - k, q);
    if (k == 0) Xk.y = 0.f;
    cplx<float>* z = buf + q * sh.S;
    const cplx<float> w = twN[k];
    z[phi_slot(sh, k)] = c2r_pre(Xk, Xc, w);
    if (k > 0 && 2 * k < H)  // exp(-2 pi i (H - k) / N) = -conj(w)
      z[phi_slot(sh, H - k)] = c2r_pre(Xc, Xk, cplx<float>{-w.x, w.y});
  }
  __syncthreads();
  phi_inverse(buf, nrow, sh, tw1);
  // one warp per row; lanes take consecutive complex points n = p + A s < A B
  const int lane = tid & 31, AB = sh.A * sh.B;
  for (int q = tid >> 5; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    double2* dst = reinterpret_cast<double2*>(a.out[f] + ((int64_t)b * nt + row) * N);
    for (int n = lane; n < AB; n += 32) {
      const int s = sh.divA(n), p = n - s * sh.A;
      const cplx<float>* z = buf + q * sh.S + p * sh.P + s;
      const cplx<float> x = z[0];
      if (sh.F == 2) {
        const cplx<float> y = z[sh.B];
        dst[n] = make_double2((double)(x.x + y.x), (double)(x.y + y.y));
        dst[n + AB] = make_double2((double)(x.x - y.x), (double)(x.y - y.y));
      } else {
        dst[n] = make_double2((double)x.x, (double)x.y);
      }
    }
  }
}

template <class SH>
__global__ void __launch_bounds__(kPhiThreads, SH::kMax <= 12 ? 4 : 3)
    k_split_to_fourier(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const SH sh(t);
  const int H = sh.H, N = 2 * H, M = t.n_m, nt = t.n_theta, tid = threadIdx.x;
  const int row = blockIdx.x, j = row >> 1;
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  cplx<float>* tw1 = buf + kPhiRows * sh.S;
  cplx<float>* twN = tw1 + (sh.A - 1) * sh.Ns;
  phi_twiddles_to_smem(tw1, sh, t);
  const int lane = tid & 31, AB = sh.A * sh.B;
  for (int q = tid >> 5; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const double2* src = reinterpret_cast<const double2*>(a.in[f] + ((int64_t)b * nt + row) * N);
#pragma unroll 4
    for (int n = lane; n < AB; n += 32) {
      const int s = sh.divA(n), p = n - s * sh.A;
      cplx<float>* z = buf + q * sh.S + p * sh.P + s;
      const double2 v = __ldg(src + n);
      const cplx<float> x = {(float)v.x, (float)v.y};
      if (sh.F == 2) {
        const double2 u = __ldg(src + n + AB);
        const cplx<float> y = {(float)u.x, (float)u.y};
        z[0] = cadd(x, y);
        z[sh.B] = csub(x, y);
      } else {
        z[0] = x;
      }
    }
  }
  __syncthreads();
  phi_forward(buf, nrow, sh, tw1);
  const float ws = (float)(t.wq[row] / N), wv = (float)(t.wq_v[row] / N);
  float* G = a.G + (int64_t)(row & 1) * a.g_h + (int64_t)j * a.g_j;
  const float rcp = 1.0f / (float)nrow;
#pragma unroll 4
  for (int e = tid; e < M * nrow; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const cplx<float>* z = buf + q * sh.S;
    const cplx<float> X = r2c_post(z[phi_slot(sh, k)], z[phi_slot(sh, k ? H - k : 0)], twN[k]);
    const float w = (a.vector_mask >> f) & 1 ? wv : ws;
    reinterpret_cast<float2*>(G + k * a.g_m + (int64_t)b * a.g_level)[f] =
        make_float2(w * X.x, w * X.y);
  }
}

// Few transforms of 25 or 27 points: block-wide Stockham passes of radices up to 8
// (fft.cuh, kStRows rows at a time through a scratch buffer).  Such a transform is a
// long chain for one thread, and a step of few leaves most threads idle; passes of
// radix 5 and 3 share the work among more.
constexpr int kStRows = 7;

__global__ void __launch_bounds__(kPhiThreads) k_split_to_grid_st(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const int N = t.n_phi, H = N / 2, M = t.n_m, nt = t.n_theta, S = padded_len(H);
  const int row = blockIdx.x, j = row >> 1, tid = threadIdx.x;
  const float hs = (row & 1) ? -1.f : 1.f;  // north = sym + asym, south = sym - asym
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  cplx<float>* tws = buf + (kPhiRows + kStRows) * S;
  fft_twiddles_to_smem(tws, H, t.twiddle, t.fft_radix, t.fft_nstages);
  const float* fs = a.Fs + (int64_t)j * a.fs_j + 2 * r0;
  const float rcp = 1.0f / (float)nrow;
  for (int e = tid; e < nrow * M; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    const float2 sy = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m) + q);
    const float2 as = __ldg(reinterpret_cast<const float2*>(fs + k * a.fs_m + a.fs_c) + q);
    buf[q * S + pad16(k)] = {sy.x + hs * as.x, sy.y + hs * as.y};
  }
  for (int e = tid; e < nrow * (H - M); e += kPhiThreads) {
    const int q = e / (H - M), k = M + e % (H - M);
    buf[q * S + pad16(k)] = {0.f, 0.f};
  }
  __syncthreads();
  // half spectrum -> Z in place (fft.cuh, c2r_pre), then the block FFT
  for (int e = tid; e < nrow * (H / 2 + 1); e += kPhiThreads) {
    const int q = e / (H / 2 + 1), k = e % (H / 2 + 1);
    cplx<float>* rw = buf + q * S;
    const int kc = H - k;
    cplx<float> Xk = rw[pad16(k)];
    if (k == 0) {
      Xk.y = 0.f;
      rw[pad16(0)] = c2r_pre(Xk, cplx<float>{0.f, 0.f}, 0, t.twiddle);
    } else {
      const cplx<float> Xc = rw[pad16(kc)];
      const cplx<float> Zk = c2r_pre(Xk, Xc, k, t.twiddle);
      const cplx<float> Zc = c2r_pre(Xc, Xk, kc, t.twiddle);
      rw[pad16(k)] = Zk;
      if (kc != k) rw[pad16(kc)] = Zc;
    }
  }
  __syncthreads();
  fft_rows<true>(buf, buf + kPhiRows * S, nrow, kStRows, H, S, t.fft_radix, t.fft_nstages, tws);
  __syncthreads();
  const int lane = tid & 31;
  for (int q = tid >> 5; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    double2* dst = reinterpret_cast<double2*>(a.out[f] + ((int64_t)b * nt + row) * N);
    for (int n = lane; n < H; n += 32) {
      const cplx<float> z = buf[q * S + pad16(n)];
      dst[n] = make_double2((double)z.x, (double)z.y);
    }
  }
}

__global__ void __launch_bounds__(kPhiThreads) k_split_to_fourier_st(SplitPhiArgs a) {
  extern __shared__ __align__(16) float smemf[];
  cplx<float>* buf = reinterpret_cast<cplx<float>*>(smemf);
  const Tables& t = a.t;
  const int N = t.n_phi, H = N / 2, M = t.n_m, nt = t.n_theta, S = padded_len(H);
  const int row = blockIdx.x, j = row >> 1, tid = threadIdx.x, lane = tid & 31;
  const int r0 = blockIdx.y * kPhiRows, nrow = min(kPhiRows, a.nrows - r0);
  cplx<float>* tws = buf + (kPhiRows + kStRows) * S;
  fft_twiddles_to_smem(tws, H, t.twiddle, t.fft_radix, t.fft_nstages);
  for (int q = tid >> 5; q < nrow; q += kPhiThreads / 32) {
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const double2* src = reinterpret_cast<const double2*>(a.in[f] + ((int64_t)b * nt + row) * N);
    for (int n = lane; n < H; n += 32) {
      const double2 v = __ldg(src + n);
      buf[q * S + pad16(n)] = {(float)v.x, (float)v.y};
    }
  }
  __syncthreads();
  fft_rows<false>(buf, buf + kPhiRows * S, nrow, kStRows, H, S, t.fft_radix, t.fft_nstages, tws);
  __syncthreads();
  const float ws = (float)(t.wq[row] / N), wv = (float)(t.wq_v[row] / N);
  float* G = a.G + (int64_t)(row & 1) * a.g_h + (int64_t)j * a.g_j;
  const float rcp = 1.0f / (float)nrow;
  for (int e = tid; e < M * nrow; e += kPhiThreads) {
    const int k = fdiv(e, rcp), q = e - k * nrow;
    const int r = r0 + q, b = r / a.nf, f = r - b * a.nf;
    const cplx<float>* z = buf + q * S;
    const cplx<float> X = r2c_post(z[pad16(k)], z[pad16((H - k) % H)], k, t.twiddle);
    const float w = (a.vector_mask >> f) & 1 ? wv : ws;
    reinterpret_cast<float2*>(G + k * a.g_m + (int64_t)b * a.g_level)[f] =
        make_float2(w * X.x, w * X.y);
  }
}

template <typename K>
static int launch_phi(K kern, size_t n_cplx, const SplitPhiArgs& a, cudaStream_t st) {
  const size_t sm = n_cplx * sizeof(cplx<float>);
  const dim3 grid(a.t.n_theta, (a.nrows + kPhiRows - 1) / kPhiRows);
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  kern<<<grid, kPhiThreads, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <int Q>
static int launch_hw(bool to_grid, const SplitPhiArgs& a, cudaStream_t st) {
  const size_t n = (size_t)kPhiRows * (16 * Q + 1) + 15 * Q + 16 * Q;
  return to_grid ? launch_phi(k_split_to_grid_hw<Q>, n, a, st)
                 : launch_phi(k_split_to_fourier_hw<Q>, n, a, st);
}

template <class SH>
static int launch_rows(bool to_grid, const SplitPhiArgs& a, cudaStream_t st) {
  const size_t n = (size_t)kPhiRows * phi_row_len(a.t) + phi_tw_len(a.t);
  return to_grid ? launch_phi(k_split_to_grid<SH>, n, a, st)
                 : launch_phi(k_split_to_fourier<SH>, n, a, st);
}

static int launch_st(bool to_grid, const SplitPhiArgs& a, cudaStream_t st) {
  const int H = a.t.n_phi / 2;
  const size_t n = (size_t)(kPhiRows + kStRows) * padded_len(H) + H;
  return launch_phi(to_grid ? k_split_to_grid_st : k_split_to_fourier_st, n, a, st);
}

int launch_split_phi(bool to_grid, const SplitPhiArgs& a, cudaStream_t st) {
  switch (a.t.n_phi) {
    case 256: return launch_hw<8>(to_grid, a, st);
    case 384: return launch_hw<12>(to_grid, a, st);
    case 512: return launch_hw<16>(to_grid, a, st);
    case 768: return launch_hw<24>(to_grid, a, st);
    default: break;
  }
  const int r = phi_max_radix(a.t);
  // Radix 25 or 27 (n_phi 250, 486, 500, 750, 800, 810, 972, 1000).  On at most eight
  // rows passes take scal_to_spat from 138 to 128 us (n_phi 1000, 1 column), from 86 to 77
  // (750), from 95 to 88 (486, l_max 324, minc 2, 8 columns); with more rows a round of
  // the four transforms takes 740 us in two steps and 819 in passes (n_phi 800, l_max
  // 266, 30 columns), 1190 and 1328 (1000, l_max 333).  With an inner step of five
  // points (250 and 500) a row is at most ten 25-point transforms, and three passes are as
  // short as two steps at any number: 301 us in passes and 333 in steps (250, l_max
  // 327, 7 columns), 276 and 285 (500, l_max 163, 14).
  if (r > 18 && (a.nrows <= 8 || a.t.fft_b <= 5)) return launch_st(to_grid, a, st);
  return r <= 12 ? launch_rows<PhiShapeRt<12>>(to_grid, a, st)
                 : launch_rows<PhiShapeRt<27>>(to_grid, a, st);
}

}  // namespace mt
