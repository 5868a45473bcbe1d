// phi stage of the drop-in transforms: Fourier rows <-> grid rows.
//
// Every grid row is one real field: synthesis is irfft(norm="forward")
// (unnormalised, Im of mode 0 ignored), analysis rfft(norm="forward"), both
// through a half-length complex FFT in shared memory (phi_fft.cuh).  Analysis
// outputs are scaled by 1/N and by the row's quadrature weight (2 pi w, or
// 2 pi w/sin^2 for vector components), so the Legendre analysis needs only P
// and dP.
#include "fourier.cuh"
#include "phi_fft.cuh"

namespace mt {

constexpr int kColsPerCta = 8;  // real columns (grid rows) per CTA

// Threads of a CTA: 256; 128, and so twice the CTAs an SM, for the largest
// radices on at most kFewCols columns, where a step has too few transforms for
// 256 threads (n_phi 250, 3 columns: 75 and 15) and the registers of a radix-25
// transform allow two CTAs of that size only: a round trip of 3 columns at l_max
// 327, minc 4 takes 173 us with 256 threads, 165 with 128.  Up to two CTAs an SM
// (kFewRows theta rows) those get all the registers they ask for instead of a
// quarter of the SM's, and the radix-25 and 27 transforms don't spill: 1 column at
// n_phi 500, l_max 166, analysis 20.9 -> 18.9 us, synthesis 20.0 -> 18.0; above, the
// limit is the better (n_phi 750, l_max 250: 26 against 29 us).
constexpr int kFftThreads = 256, kFewThreads = 128, kFewCols = 4, kFewRows = 2 * kSms;

constexpr int fft_ctas(int kMax) { return kMax <= 12 ? 3 : 2; }

template <class SH, int T, int kCtas>
__global__ void __launch_bounds__(T, kCtas) k_fourier_to_grid(ToGridArgs a) {
  extern __shared__ double smem[];
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem);
  const Tables& t = a.t;
  const SH sh(t);
  const int H = sh.H, N = 2 * H, M = t.n_m, nt = t.n_theta;
  const int row = blockIdx.y;
  const int col0 = blockIdx.x * kColsPerCta;
  const int ncol = min(kColsPerCta, a.ncols - col0);
  cplx<double>* tw1 = buf + kColsPerCta * sh.S;
  cplx<double>* twN = tw1 + (sh.A - 1) * sh.Ns;
  phi_twiddles_to_smem(tw1, sh, t);
  const double2* Fr = a.F + (int64_t)row * a.f_row + col0;
  const float rcp = 1.0f / (float)ncol;
  // pairs (k, H - k) of every column: Z[k] = c2r_pre(X[k], X[H - k]) with X = 0
  // at k >= M (and X[H] = 0: 2 (n_m - 1) < N), kLd pairs in flight per thread
  constexpr int kLd = 4;
  const int total = (H / 2 + 1) * ncol;
  for (int e0 = 0; e0 < total; e0 += kLd * T) {
    double2 xa[kLd], xb[kLd];
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int e = e0 + u * T + threadIdx.x, k = fdiv(e, rcp), q = e - k * ncol;
      xa[u] = xb[u] = make_double2(0.0, 0.0);
      if (e < total) {
        if (k < M) xa[u] = __ldg(&Fr[k * a.f_m + q]);
        if (k > 0 && H - k < M) xb[u] = __ldg(&Fr[(H - k) * a.f_m + q]);
      }
    }
    if (e0 == 0) {  // the tables are complete once every thread's copies are
      cp_async_wait_all();
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int e = e0 + u * T + threadIdx.x, k = fdiv(e, rcp), q = e - k * ncol;
      if (e < total) {
        cplx<double>* z = buf + q * sh.S;
        const cplx<double> w = twN[k];
        const cplx<double> Xk = {xa[u].x, k ? xa[u].y : 0.0}, Xc = {xb[u].x, xb[u].y};
        z[phi_slot(sh, k)] = c2r_pre(Xk, Xc, w);
        if (k > 0 && 2 * k < H)  // exp(-2 pi i (H - k) / N) = -conj(w)
          z[phi_slot(sh, H - k)] = c2r_pre(Xc, Xk, cplx<double>{-w.x, w.y});
      }
    }
  }
  __syncthreads();
  phi_inverse(buf, ncol, sh, tw1);
  // one warp per row; lanes take consecutive complex points n = p + A s < A B
  const int lane = threadIdx.x & 31, AB = sh.A * sh.B;
  for (int q = threadIdx.x >> 5; q < ncol; q += T / 32) {
    const int c = col0 + q, f = c / a.B, b = c - f * a.B;
    double* dst = a.out[f] + ((int64_t)b * nt + row) * N;
    const bool wide = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    auto put = [&](int n, double x, double y) {
      if (wide) reinterpret_cast<double2*>(dst)[n] = make_double2(x, y);
      else {
        dst[2 * n] = x;
        dst[2 * n + 1] = y;
      }
    };
    for (int n = lane; n < AB; n += 32) {
      const int s = sh.divA(n), p = n - s * sh.A;
      const cplx<double>* z = buf + q * sh.S + p * sh.P + s;
      const cplx<double> x = z[0];
      if (sh.F == 2) {
        const cplx<double> y = z[sh.B];
        put(n, x.x + y.x, x.y + y.y);
        put(n + AB, x.x - y.x, x.y - y.y);
      } else {
        put(n, x.x, x.y);
      }
    }
  }
}

template <class SH, int T, int kCtas>
__global__ void __launch_bounds__(T, kCtas) k_grid_to_fourier(ToFourierArgs a) {
  extern __shared__ double smem[];
  cplx<double>* buf = reinterpret_cast<cplx<double>*>(smem);
  const Tables& t = a.t;
  const SH sh(t);
  const int H = sh.H, N = 2 * H, M = t.n_m, nt = t.n_theta;
  const int row = blockIdx.y;
  const int col0 = blockIdx.x * kColsPerCta;
  const int ncol = min(kColsPerCta, a.ncols - col0);
  cplx<double>* tw1 = buf + kColsPerCta * sh.S;
  cplx<double>* twN = tw1 + (sh.A - 1) * sh.Ns;
  phi_twiddles_to_smem(tw1, sh, t);
  const int lane = threadIdx.x & 31, AB = sh.A * sh.B;
  for (int q = threadIdx.x >> 5; q < ncol; q += T / 32) {
    const int c = col0 + q, f = c / a.B, b = c - f * a.B;
    const double2* src =
        reinterpret_cast<const double2*>(a.in[f] + ((int64_t)b * nt + row) * N);
#pragma unroll 4
    for (int n = lane; n < AB; n += 32) {
      const int s = sh.divA(n), p = n - s * sh.A;
      cplx<double>* z = buf + q * sh.S + p * sh.P + s;
      const double2 x = __ldg(&src[n]);
      if (sh.F == 2) {
        const double2 y = __ldg(&src[n + AB]);
        z[0] = {x.x + y.x, x.y + y.y};
        z[sh.B] = {x.x - y.x, x.y - y.y};
      } else {
        z[0] = {x.x, x.y};
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();
  phi_forward(buf, ncol, sh, tw1);
  const double w = (a.vector ? t.wq_v[row] : t.wq[row]) / N;
  double2* Fr = a.F + (int64_t)row * a.f_row + col0;
  const float rcpc = 1.0f / (float)ncol;
#pragma unroll 4
  for (int e = threadIdx.x; e < M * ncol; e += T) {
    const int k = fdiv(e, rcpc), q = e - k * ncol;
    const cplx<double>* z = buf + q * sh.S;
    const cplx<double> X = r2c_post(z[phi_slot(sh, k)], z[phi_slot(sh, k ? H - k : 0)], twN[k]);
    Fr[k * a.f_m + q] = make_double2(w * X.x, w * X.y);
  }
}

static size_t fft_smem(const Tables& t) {
  return ((size_t)kColsPerCta * phi_row_len(t) + phi_tw_len(t)) * sizeof(double2);
}

template <int kMax, int T = kFftThreads, int kCtas = fft_ctas(kMax)>
static int launch_to_grid(const ToGridArgs& a, cudaStream_t st) {
  const size_t sm = fft_smem(a.t);
  auto kern = k_fourier_to_grid<PhiShapeRt<kMax>, T, kCtas>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  dim3 grid((a.ncols + kColsPerCta - 1) / kColsPerCta, a.t.n_theta);
  kern<<<grid, T, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <int kMax, int T = kFftThreads, int kCtas = fft_ctas(kMax)>
static int launch_to_fourier(const ToFourierArgs& a, cudaStream_t st) {
  const size_t sm = fft_smem(a.t);
  auto kern = k_grid_to_fourier<PhiShapeRt<kMax>, T, kCtas>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  dim3 grid((a.ncols + kColsPerCta - 1) / kColsPerCta, a.t.n_theta);
  kern<<<grid, T, sm, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

int launch_fourier_to_grid(const ToGridArgs& a, cudaStream_t st) {
  const int r = phi_max_radix(a.t);
  if (r <= 12) return launch_to_grid<12>(a, st);
  if (r <= 18) return launch_to_grid<18>(a, st);
  if (a.ncols > kFewCols) return launch_to_grid<27>(a, st);
  return a.t.n_theta <= kFewRows ? launch_to_grid<27, kFewThreads, 2>(a, st)
                                 : launch_to_grid<27, kFewThreads, 4>(a, st);
}

int launch_grid_to_fourier(const ToFourierArgs& a, cudaStream_t st) {
  const int r = phi_max_radix(a.t);
  if (r <= 12) return launch_to_fourier<12>(a, st);
  if (r <= 18) return launch_to_fourier<18>(a, st);
  if (a.ncols > kFewCols) return launch_to_fourier<27>(a, st);
  return a.t.n_theta <= kFewRows ? launch_to_fourier<27, kFewThreads, 2>(a, st)
                                 : launch_to_fourier<27, kFewThreads, 4>(a, st);
}

// Largest n_phi that the row FFTs' two radices cover (phi_fft.cuh).
int fft_max_nphi() { return 1168; }

}  // namespace mt
