// Row FFTs of the phi stage, in place in shared memory.
//
// A real row of length N = n_phi goes through a complex FFT of half length
// H = N/2 (c2r_pre / r2c_post, fft.cuh), factored H = A B F, F = 2 for even H
// (1 for odd).  The inverse (synthesis) runs decimation in frequency: an outer
// step of A-point DFTs, an inner step of B-point DFTs, then the F-point
// butterflies; the forward (analysis) runs the transposed chain, decimation in
// time, F, B, A.  Every step works in place, so wavenumbers are in natural
// order on both ends and the grid points in between are permuted:
//   element (p, s, g), p < A, s < B, g < F, is complex point n = p + A (s + B g)
//   (grid points 2 n and 2 n + 1).
// A stage that is pointwise in phi takes the points as they lie and does the
// F = 2 butterfly on its own operands: it is a plain sum and difference, the
// same for real and imaginary parts.  So a row crosses shared memory three
// times each way (coefficients in, outer step, inner step), against five for a
// chain of radix-12, 4, 4, 2 passes: shared memory is what bounds the phi
// kernels (its pipe was 60 % busy at n_phi = 768).  Measured against the passes
// replaced: the FP64 Boussinesq phi stage at l_max 255 on 97 levels (n_phi 768,
// warp FFTs) 2.74 -> 2.33 ms, the anelastic one at l_max 383 on 129 levels
// (n_phi 1152, radix-8/3 stages) 9.16 -> 5.8 ms, the FP64 transforms of 37 columns
// at l_max 213 (n_phi 640, out-of-place Stockham passes) 1.00 -> 0.73 ms in all.
// Shared memory is 55 % busy now, the FP64 pipe 36 %, at 16 warps an SM.
//
// Layout of a row: element (p, f, q) of wavenumber k = p F B + F q + f (outer
// and inner step inputs) or of point (p, s = q, g = f) sits at
//   p P + f B + q,  P = F B | 1.
// The odd block stride P makes the inner step and the butterflies (lanes on
// consecutive p) free of bank conflicts when A is a multiple of 8, the odd row
// stride S nearly so the load and store phases (lanes on consecutive fields of
// one k); the outer step reads runs of consecutive slots.
//
// Radices (2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 25, 27) cover every H with
// factors 2, 3, 5 up to 584 in the two steps; phi_factor (tables.cu) picks the
// pair.
#pragma once

#include "fft.cuh"

namespace mt {

// cos and sin of 2 pi e / N, 0 <= e <= N / 2, e a constant after unrolling.
template <int N>
__device__ __forceinline__ double2 phi_cs(int e) {
  if constexpr (N == 15) {
    static constexpr double c[] = {1.0, 0.9135454576426009, 0.6691306063588582, 0.30901699437494745,
        -0.10452846326765347, -0.5, -0.8090169943749475, -0.9781476007338057};
    static constexpr double s[] = {0.0, 0.4067366430758002, 0.7431448254773942, 0.9510565162951535,
        0.9945218953682733, 0.8660254037844386, 0.5877852522924731, 0.20791169081775934};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 24) {
    static constexpr double c[] = {1.0, 0.9659258262890683, 0.8660254037844386, 0.7071067811865476,
        0.5, 0.25881904510252074, 0.0, -0.25881904510252074, -0.5, -0.7071067811865476,
        -0.8660254037844386, -0.9659258262890683, -1.0};
    static constexpr double s[] = {0.0, 0.25881904510252074, 0.5, 0.7071067811865476,
        0.8660254037844386, 0.9659258262890683, 1.0, 0.9659258262890683, 0.8660254037844386,
        0.7071067811865476, 0.5, 0.25881904510252074, 0.0};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 25) {
    static constexpr double c[] = {1.0, 0.9685831611286311, 0.8763066800438636, 0.7289686274214116,
        0.5358267949789967, 0.30901699437494745, 0.06279051952931337, -0.18738131458572463,
        -0.42577929156507266, -0.6374239897486897, -0.8090169943749475, -0.9297764858882515,
        -0.9921147013144779};
    static constexpr double s[] = {0.0, 0.2486898871648548, 0.48175367410171527, 0.6845471059286887,
        0.8443279255020151, 0.9510565162951535, 0.9980267284282716, 0.9822872507286887,
        0.9048270524660196, 0.7705132427757893, 0.5877852522924731, 0.368124552684678,
        0.12533323356430426};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 27) {
    static constexpr double c[] = {1.0, 0.9730448705798238, 0.8936326403234123, 0.766044443118978,
        0.5971585917027862, 0.39607976603915684, 0.17364817766693036, -0.05814482891047583,
        -0.28680323271109026, -0.5, -0.6862416378687336, -0.8354878114129364, -0.9396926207859084,
        -0.993238357741943};
    static constexpr double s[] = {0.0, 0.23061587074244017, 0.44879918020046217,
        0.6427876096865394, 0.8021231927550437, 0.918216106880274, 0.984807753012208,
        0.9983081582712682, 0.9579895123154889, 0.8660254037844386, 0.7273736415730487,
        0.549508978070806, 0.3420201433256687, 0.11609291412523023};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 32) {
    static constexpr double c[] = {1.0, 0.9807852804032304, 0.9238795325112867, 0.8314696123025452,
        0.7071067811865476, 0.5555702330196022, 0.3826834323650898, 0.19509032201612828, 0.0,
        -0.19509032201612828, -0.3826834323650898, -0.5555702330196022, -0.7071067811865476,
        -0.8314696123025452, -0.9238795325112867, -0.9807852804032304, -1.0};
    static constexpr double s[] = {0.0, 0.19509032201612828, 0.3826834323650898, 0.5555702330196022,
        0.7071067811865476, 0.8314696123025452, 0.9238795325112867, 0.9807852804032304, 1.0,
        0.9807852804032304, 0.9238795325112867, 0.8314696123025452, 0.7071067811865476,
        0.5555702330196022, 0.3826834323650898, 0.19509032201612828, 0.0};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 36) {
    static constexpr double c[] = {1.0, 0.984807753012208, 0.9396926207859084, 0.8660254037844386,
        0.766044443118978, 0.6427876096865394, 0.5, 0.3420201433256687, 0.17364817766693036, 0.0,
        -0.17364817766693036, -0.3420201433256687, -0.5, -0.6427876096865394, -0.766044443118978,
        -0.8660254037844386, -0.9396926207859084, -0.984807753012208, -1.0};
    static constexpr double s[] = {0.0, 0.17364817766693036, 0.3420201433256687, 0.5,
        0.6427876096865394, 0.766044443118978, 0.8660254037844386, 0.9396926207859084,
        0.984807753012208, 1.0, 0.984807753012208, 0.9396926207859084, 0.8660254037844386,
        0.766044443118978, 0.6427876096865394, 0.5, 0.3420201433256687, 0.17364817766693036, 0.0};
    return make_double2(c[e], s[e]);
  } else if constexpr (N == 40) {
    static constexpr double c[] = {1.0, 0.9876883405951378, 0.9510565162951535, 0.8910065241883679,
        0.8090169943749475, 0.7071067811865476, 0.5877852522924731, 0.4539904997395468,
        0.30901699437494745, 0.15643446504023087, 0.0, -0.15643446504023087, -0.30901699437494745,
        -0.4539904997395468, -0.5877852522924731, -0.7071067811865476, -0.8090169943749475,
        -0.8910065241883679, -0.9510565162951535, -0.9876883405951378, -1.0};
    static constexpr double s[] = {0.0, 0.15643446504023087, 0.30901699437494745,
        0.4539904997395468, 0.5877852522924731, 0.7071067811865476, 0.8090169943749475,
        0.8910065241883679, 0.9510565162951535, 0.9876883405951378, 1.0, 0.9876883405951378,
        0.9510565162951535, 0.8910065241883679, 0.8090169943749475, 0.7071067811865476,
        0.5877852522924731, 0.4539904997395468, 0.30901699437494745, 0.15643446504023087, 0.0};
    return make_double2(c[e], s[e]);
  }
}

// exp(-+ 2 pi i e / N) (forward -, inverse +), e a constant after unrolling, N
// a radix or twice one: read from the table of a multiple of N.
template <int N, bool INV, typename T>
__device__ __forceinline__ cplx<T> phi_root(int e) {
  constexpr int M = 24 % N == 0   ? 24
                    : 32 % N == 0 ? 32
                    : 36 % N == 0 ? 36
                    : 40 % N == 0 ? 40
                    : 15 % N == 0 ? 15
                    : N % 27 == 0 ? 27
                    : N % 25 == 0 ? 25
                                  : 15;
  bool neg = false;
  if (M % N != 0) {  // N = 2 M, M odd: w_N^e = w_M^(e / 2), or -w_M^((e + M) / 2)
    neg = e % 2 != 0;
    e = (neg ? e + M : e) / 2;
  } else {
    e = e * (M / N);
  }
  e %= M;
  const bool up = 2 * e > M;  // the lower half circle by conjugation
  const double2 w = phi_cs<M>(up ? M - e : e);
  double c = w.x, s = up ? -w.y : w.y;
  if (neg) {
    c = -c;
    s = -s;
  }
  return {(T)c, (T)(INV ? s : -s)};
}

// v times that root.
template <int N, bool INV, typename T>
__device__ __forceinline__ cplx<T> phi_rot(cplx<T> v, int e) {
  if (e == 0) return v;
  if (4 * e == N) return mul_mi<INV>(v);
  if (2 * e == N) return {-v.x, -v.y};
  return cmul(v, phi_root<N, INV, T>(e));
}

// R-point DFT in registers: R = R1 R2, n = R2 a + b, k = k1 + R1 k2.
template <int R, bool INV, typename T>
__device__ __forceinline__ void phi_dft(cplx<T> (&v)[R]) {
  if constexpr (R == 2 || R == 3 || R == 4 || R == 5 || R == 8 || R == 16) {
    dft_small<R, INV>(v);
  } else {
    constexpr int R2 = R % 5 == 0 && R != 15 ? 5 : 3, R1 = R / R2;
    cplx<T> t[R2][R1];
#pragma unroll
    for (int b = 0; b < R2; ++b) {
      cplx<T> u[R1];
#pragma unroll
      for (int a = 0; a < R1; ++a) u[a] = v[R2 * a + b];
      phi_dft<R1, INV>(u);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) t[b][k1] = phi_rot<R, INV>(u[k1], b * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      cplx<T> u[R2];
#pragma unroll
      for (int b = 0; b < R2; ++b) u[b] = t[b][k1];
      phi_dft<R2, INV>(u);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = u[k2];
    }
  }
}

// Shape of the rows, compile-time or from the plan.  The run-time one compiles
// the radices up to kMax only: a kernel's registers follow its largest radix.
template <int A_, int B_, int F_>
struct PhiShape {
  static constexpr bool kStatic = true;
  __device__ explicit PhiShape(const Tables&) {}
  static constexpr int A = A_, B = B_, F = F_, Ns = F * B, P = Ns | 1, S = (A * P) | 1,
                       H = A * Ns;
  __device__ static int divNs(int i) { return i / Ns; }
  __device__ static int divFA(int i) { return i / (F * A); }
  __device__ static int divB(int i) { return i / B; }
  __device__ static int divA(int i) { return i / A; }
};
template <int kMax_>
struct PhiShapeRt {
  static constexpr bool kStatic = false;
  static constexpr int kMax = kMax_;
  int A, B, F, Ns, P, S, H;
  float rNs, rFA, rB, rA;
  __device__ explicit PhiShapeRt(const Tables& t) {
    A = t.fft_a;
    B = t.fft_b;
    F = t.fft_f;
    Ns = F * B;
    P = Ns | 1;
    S = (A * P) | 1;
    H = A * Ns;
    rNs = 1.0f / (float)Ns;
    rFA = 1.0f / (float)(F * A);
    rB = 1.0f / (float)B;
    rA = 1.0f / (float)A;
  }
  __device__ int divNs(int i) const { return fdiv(i, rNs); }
  __device__ int divFA(int i) const { return fdiv(i, rFA); }
  __device__ int divB(int i) const { return fdiv(i, rB); }
  __device__ int divA(int i) const { return fdiv(i, rA); }
};

// Slot of wavenumber k in a row.
template <class SH>
__device__ __forceinline__ int phi_slot(const SH& sh, int k) {
  const int p = sh.divNs(k), j = k - p * sh.Ns;
  return p * sh.P + (sh.F == 2 ? (j & 1) * sh.B + (j >> 1) : j);
}

// Outer step: A-point DFTs over p of every slot of a block.
// tw1[(q - 1) Ns + slot] = exp(-2 pi i q j / H), j the wavenumber of the slot.
template <int R, bool INV, class SH, typename T>
__device__ __forceinline__ void phi_outer_r(cplx<T>* buf, int nrows, const SH& sh,
                                            const cplx<T>* __restrict__ tw1) {
  const int total = nrows * sh.Ns;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int row = sh.divNs(it), j = it - row * sh.Ns;
    cplx<T>* x = buf + row * sh.S + j;
    cplx<T> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[q * sh.P];
    if (INV) phi_dft<R, INV>(v);
    // w^q, w = tw1's exp(-2 pi i j / H): in FP64 read for q < 4 and multiples of
    // four, one product (one rounding) for the others, 6 of 15 reads at R = 16;
    // in FP32, where that rounding would show and the reads are half the size,
    // all read
    cplx<T> wb[4];
#pragma unroll
    for (int q = 1; q < R; ++q) {
      cplx<T> w;
      if (sizeof(T) == 4 || q < 4 || q % 4 == 0) {
        w = tw1[(q - 1) * sh.Ns + j];
        if (INV) w.y = -w.y;
        if (q < 4) wb[q] = w;
        else if (q % 4 == 0) wb[0] = w;
      } else {
        w = cmul(wb[0], wb[q % 4]);
      }
      v[q] = cmul(v[q], w);
    }
    if (!INV) phi_dft<R, INV>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) x[q * sh.P] = v[q];
  }
}

// Inner step: B-point DFTs over the contiguous runs (p, f) of a block; the
// twiddles between it and the F = 2 butterfly are exp(-2 pi i s / (2 B)) on
// the runs f = 1 (lanes of one warp mostly share f).
template <int R, bool INV, class SH, typename T>
__device__ __forceinline__ void phi_inner_r(cplx<T>* buf, int nrows, const SH& sh) {
  const int FA = sh.F * sh.A, total = nrows * FA;
  for (int it = threadIdx.x; it < total; it += blockDim.x) {
    const int row = sh.divFA(it), u = it - row * FA;
    const int f = u >= sh.A, p = u - (f ? sh.A : 0);
    cplx<T>* x = buf + row * sh.S + p * sh.P + f * sh.B;
    cplx<T> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[q];
    if (INV) phi_dft<R, INV>(v);
    if (f) {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = phi_rot<2 * R, INV>(v[q], q);
    }
    if (!INV) phi_dft<R, INV>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = v[q];
  }
}

#define MT_PHI_RADICES(X) \
  X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16) X(18) X(25) X(27)

template <bool INV, class SH, typename T>
__device__ __forceinline__ void phi_outer(cplx<T>* buf, int nrows, const SH& sh,
                                          const cplx<T>* __restrict__ tw1) {
  if constexpr (SH::kStatic) {
    phi_outer_r<SH::A, INV>(buf, nrows, sh, tw1);
  } else {
    switch (sh.A) {
#define X(r)                                                                     \
  case r:                                                                        \
    if constexpr (r <= SH::kMax) phi_outer_r<r, INV>(buf, nrows, sh, tw1);       \
    break;
      MT_PHI_RADICES(X)
#undef X
      default: break;  // A = 1: nothing to do
    }
  }
  __syncthreads();
}

template <bool INV, class SH, typename T>
__device__ __forceinline__ void phi_inner(cplx<T>* buf, int nrows, const SH& sh) {
  if constexpr (SH::kStatic) {
    phi_inner_r<SH::B, INV>(buf, nrows, sh);
  } else {
    switch (sh.B) {
#define X(r)                                                                     \
  case r:                                                                        \
    if constexpr (r <= SH::kMax) phi_inner_r<r, INV>(buf, nrows, sh);            \
    break;
      MT_PHI_RADICES(X)
#undef X
      default: break;
    }
  }
  __syncthreads();
}

// Inverse transforms up to the F butterflies, forward ones from behind them.
template <class SH, typename T>
__device__ __forceinline__ void phi_inverse(cplx<T>* buf, int nrows, const SH& sh,
                                            const cplx<T>* tw1) {
  phi_outer<true>(buf, nrows, sh, tw1);
  phi_inner<true>(buf, nrows, sh);
}
template <class SH, typename T>
__device__ __forceinline__ void phi_forward(cplx<T>* buf, int nrows, const SH& sh,
                                            const cplx<T>* tw1) {
  phi_inner<false>(buf, nrows, sh);
  phi_outer<false>(buf, nrows, sh, tw1);
}

// The row twiddles: tw1 ((A - 1) Ns values) then twN (H values).  FP64 tables
// are copied asynchronously from the plan's (the caller waits with
// cp_async_wait_all and synchronises); FP32 ones are converted.
template <class SH>
__device__ __forceinline__ int phi_tw_len(const SH& sh) {
  return (sh.A - 1) * sh.Ns + sh.H;
}
template <class SH, typename T>
__device__ __forceinline__ void phi_twiddles_to_smem(cplx<T>* tws, const SH& sh, const Tables& t) {
  const int n1 = (sh.A - 1) * sh.Ns, n = n1 + sh.H;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double2* src = i < n1 ? &t.phi_tw1[i] : &t.twiddle[i - n1];
    if constexpr (sizeof(T) == 8) {
      cp_async16(&tws[i], src);
    } else {
      const double2 w = __ldg(src);
      tws[i] = {(T)w.x, (T)w.y};
    }
  }
}

// The phases of a fused stage around the row FFTs (T = blockDim.x threads).

// Asks the L2 for the rows of a CTA one wave further along the grid (x fastest), so
// that they are there when it takes this one's place: a wave is 512 threads an SM,
// what the stages' launch bounds ask for (where shared memory holds fewer CTAs, the
// rows wait in the L2 for longer).  at(row, r) is the address of its k = 0 entry,
// `pitch` doubles from one k to the next; the first and the last line of the NF
// complex values of one k are asked for.
template <int NF, int T, typename At>
__device__ __forceinline__ void phi_prefetch(int M, int64_t pitch, At at) {
  constexpr int kAhead = 512 / T * kSms;
  const int id = blockIdx.y * gridDim.x + blockIdx.x + kAhead;
  const int row = id / gridDim.x, r = id - row * gridDim.x;
  if (row >= (int)gridDim.y) return;
  const double* x = at(row, r);
  for (int e = threadIdx.x; e < 2 * M; e += T)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(x + (e >> 1) * pitch + (e & 1) * (2 * NF - 1)));
}

// Rows of the NF fields from their half spectra ld(k, f), k < M (zero above,
// Im of k = 0 ignored), with the real-row pre-processing of the pairs
// (k, H - k), k <= H / 2: Z[k] = c2r_pre(X[k], X[H - k]) and Z[H - k] =
// c2r_pre(X[H - k], X[k]).  kLd pairs per thread are loaded before any is
// stored, so their HBM latencies overlap (the first round's also cover the
// asynchronous copies of the twiddle tables).
template <int NF, int T, class SH, typename R, typename Ld>
__device__ __forceinline__ void phi_load_rows(cplx<R>* buf, const SH& sh, int M,
                                              const cplx<R>* __restrict__ twN, Ld ld) {
  constexpr int kLd = 6;
  const int H = sh.H, total = (H / 2 + 1) * NF;
  for (int e0 = 0; e0 < total; e0 += kLd * T) {
    cplx<R> xa[kLd], xb[kLd];
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int e = e0 + u * T + (int)threadIdx.x, k = e / NF, f = e - k * NF;
      xa[u] = xb[u] = {(R)0, (R)0};
      if (e < total) {
        if (k < M) xa[u] = ld(k, f);
        if (k > 0 && H - k < M) xb[u] = ld(H - k, f);
      }
    }
    if (e0 == 0) {  // (uniform) the tables are complete once every thread's copies are
      cp_async_wait_all();
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < kLd; ++u) {
      const int e = e0 + u * T + (int)threadIdx.x, k = e / NF, f = e - k * NF;
      if (e < total) {
        cplx<R>* z = buf + f * sh.S;
        const cplx<R> w = twN[k];
        const cplx<R> Xk = {xa[u].x, k ? xa[u].y : (R)0};
        z[phi_slot(sh, k)] = c2r_pre(Xk, xb[u], w);
        if (k > 0 && 2 * k < H)  // exp(-2 pi i (H - k) / N) = -conj(w)
          z[phi_slot(sh, H - k)] = c2r_pre(xb[u], Xk, cplx<R>{-w.x, w.y});
      }
    }
  }
  __syncthreads();
}

// point(in[NFI], out[NFO]) at every grid point, between phi_inverse and
// phi_forward: a thread takes one component (real or imaginary part) of the
// two elements g = 0, 1 of (p, s), which are two grid points after the F = 2
// butterfly, and puts the outputs' butterfly in their place.
template <int NFI, int NFO, int T, class SH, typename R, typename Fn>
__device__ __forceinline__ void phi_points(cplx<R>* buf, const SH& sh, Fn& point) {
  R* bd = reinterpret_cast<R*>(buf);
  const int total = 2 * sh.A * sh.B, S2 = 2 * sh.S, g = 2 * sh.B;
  for (int e = threadIdx.x; e < total; e += T) {
    const int u = e >> 1, s = sh.divA(u), p = u - s * sh.A;
    R* x = bd + 2 * (p * sh.P + s) + (e & 1);
    R v0[NFI], o0[NFO];
    if (sh.F == 2) {
      R v1[NFI], o1[NFO];
#pragma unroll
      for (int f = 0; f < NFI; ++f) {
        const R y0 = x[f * S2], y1 = x[f * S2 + g];
        v0[f] = y0 + y1;
        v1[f] = y0 - y1;
      }
      point(v0, o0);
      point(v1, o1);
#pragma unroll
      for (int f = 0; f < NFO; ++f) {
        x[f * S2] = o0[f] + o1[f];
        x[f * S2 + g] = o0[f] - o1[f];
      }
    } else {
#pragma unroll
      for (int f = 0; f < NFI; ++f) v0[f] = x[f * S2];
      point(v0, o0);
#pragma unroll
      for (int f = 0; f < NFO; ++f) x[f * S2] = o0[f];
    }
  }
}

// put(k, f, X[k]) for the half spectra k < M of the NF rows.
template <int NF, int T, class SH, typename R, typename Put>
__device__ __forceinline__ void phi_store_rows(const cplx<R>* buf, const SH& sh, int M,
                                               const cplx<R>* __restrict__ twN, Put put) {
  constexpr int kSt = 4;  // outputs per thread whose shared-memory reads are issued together
  for (int e0 = threadIdx.x; e0 < M * NF; e0 += kSt * T) {
    cplx<R> zk[kSt], zc[kSt], wn[kSt];
#pragma unroll
    for (int u = 0; u < kSt; ++u) {
      const int e = e0 + u * T, k = e / NF, f = e - k * NF;
      if (e < M * NF) {
        const cplx<R>* z = buf + f * sh.S;
        zk[u] = z[phi_slot(sh, k)];
        zc[u] = z[phi_slot(sh, k ? sh.H - k : 0)];
        wn[u] = twN[k];
      }
    }
#pragma unroll
    for (int u = 0; u < kSt; ++u) {
      const int e = e0 + u * T, k = e / NF, f = e - k * NF;
      if (e < M * NF) put(k, f, r2c_post(zk[u], zc[u], wn[u]));
    }
  }
}

// Shapes that the FP64 phi stages compile in: all of outer radix 16, n_phi 512, 640,
// 768, 960, 1024 and 1152, the inner radices of MT_PHI_STATIC_B.  There strides and
// divisions become constants and the radix switch goes, and with PhiShapeRt the
// Boussinesq stages take 4 to 12 % longer, the anelastic ones 3 to 7 % (65 levels,
// FP64 contractions: n_phi 512 1.91 and 2.08 ms, 768 5.53 and 5.76, 640 anelastic
// 4.20 and 4.29).  Each shape costs twelve kernels; of the lengths without one, the
// short ones have stages bound by their launches and Legendre contractions.
#define MT_PHI_STATIC_B(X) X(8) X(10) X(12) X(15) X(16) X(18)
inline bool phi_shape_static(const Tables& t) { return t.fft_a == 16 && t.fft_f == 2; }

// Largest radix, slots of a row and table entries of the plan's shape (host).
inline int phi_max_radix(const Tables& t) { return t.fft_a > t.fft_b ? t.fft_a : t.fft_b; }
inline int phi_row_len(const Tables& t) { return (t.fft_a * ((t.fft_f * t.fft_b) | 1)) | 1; }
inline int phi_tw_len(const Tables& t) { return (2 * t.fft_a - 1) * t.fft_f * t.fft_b; }

}  // namespace mt
