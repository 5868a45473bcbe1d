// FP64 Legendre contractions on the FP64 tensor pipe (mma.sync m8n8k4 f64).
//
// Synthesis, per order m (grid z), 32 northern theta (grid y) and R columns
// (grid x, fastest so that consecutive CTAs reuse the same table tile in L2):
//   K loop over l in chunks of 16 rows (8 even + 8 odd l-m); every warp owns
//   one 8-row theta tile and a column tile (two real columns a column, eight a
//   tile; two tiles for the one-term operations) and accumulates BOTH parities of
//   EVERY product of the operation, so the north/south unfolding and the
//   product combination happen in registers.
// Analysis, per order m, 64 rows l (8 warps = 8 row tiles of one parity
// each) and R columns: K loop over theta pairs in chunks of 16; the B
// operand is folded (north +/- south) according to the row parity and the
// table parity.
// Both read their chunks by asynchronous copies through a ring of buffers (as
// many as fit beside the SM's other CTAs, at most four) with one barrier a chunk.
//
// What bounds them is the FP64 tensor pipe and what the warps do between its
// instructions: a CTA's warps stage, meet and multiply in step, and the pipe
// idles while they stage.  Hence
//   * little staging work: a thread copies the same row and column of every term
//     (a copy through registers, with factors and index arithmetic, came to ten
//     instructions per tensor instruction at seven terms and eleven products);
//     l(l+1) factors and the curl's difference are taken on the fragments, by
//     operation at compile time, the fold in place by the copying thread;
//   * four CTAs of four warps an SM for the synthesis of several terms instead of
//     two of eight, so that more phases overlap (the analysis gained nothing from
//     the same split: its fold would be done twice as often).
// FP64 Boussinesq stage at l_max 170 on 65 levels: 2.16 -> 1.86 ms, at l_max 255 on
// 97 levels 7.93 -> 6.99 ms; anelastic one at l_max 127 on 65 levels 1.09 -> 0.98 ms;
// transforms of 37 columns at l_max 213 685 -> 645 us.
#include "legendre.cuh"

namespace mt {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp8(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Ring depth for a chunk of `bytes`: the CTAs of an SM keep 220 KB of chunks.
constexpr int ring_depth(int bytes, int ctas = 2) {
  return bytes * 4 * ctas <= 220 * 1024 ? 4 : bytes * 3 * ctas <= 220 * 1024 ? 3 : 2;
}

// A table tile of ROWS x COLS (rows row0 + .. < nrow, columns col0 + .. < ncol of a
// row-major table, zeros outside) into shared rows of stride S, by 16-byte copies
// where the table's rows start on 16 bytes (ncol even; col0 is), else 8-byte ones.
template <int T, int ROWS, int COLS, int S>
__device__ __forceinline__ void stage_table(double* dst, const double* __restrict__ tab, int row0,
                                            int nrow, int col0, int ncol) {
  if (ncol % 2 == 0) {
    constexpr int kRows = 2 * T / COLS;  // rows per sweep of the CTA
    const int r = threadIdx.x / (COLS / 2), j = 2 * (threadIdx.x % (COLS / 2));
#pragma unroll
    for (int i = 0; i < ROWS / kRows; ++i) {
      const int row = row0 + r + kRows * i;
      const bool ok = row < nrow && col0 + j < ncol;
      cp16(dst + (r + kRows * i) * S + j, tab + (ok ? (int64_t)row * ncol + col0 + j : 0), ok);
    }
  } else {
    constexpr int kRows = T / COLS;
    const int r = threadIdx.x / COLS, j = threadIdx.x % COLS;
#pragma unroll 1
    for (int i = 0; i < ROWS / kRows; ++i) {
      const int row = row0 + r + kRows * i;
      const bool ok = row < nrow && col0 + j < ncol;
      cp8(dst + (r + kRows * i) * S + j, tab + (ok ? (int64_t)row * ncol + col0 + j : 0), ok);
    }
  }
}

// Row strides of the staged tiles.  A fragment load reads 4 K rows x 8 columns (A
// of the synthesis, B) or 8 rows x 4 K (A of the analysis) of doubles, served by
// half-warps: four neighbours' rows must fall on different quarters of the 128
// bytes, i.e. lie 32 bytes apart mod 128.  The K rows of one parity are two apart
// in the synthesis (stride 2 mod 16 doubles, so SA = 34 and SB = 2 R + 2) and
// consecutive in the analysis's B (4 mod 16: 2 R + 4).  At 64 bytes apart, which
// took two passes, the FP64 stage at l_max 170 on 65 levels was 2.24 ms (now 2.16)
// and the transforms of 37 columns at l_max 213 0.73 ms (now 0.685); the kernels
// are bound by the FP64 tensor pipe and by these loads.
template <class OP, int R>
struct SynthCfg {
  static constexpr int TH = 32, KC = 16;
  static constexpr int SA = 34;         // sA row stride (doubles): rows 2 apart 32 mod 128 B
  static constexpr int SB = 2 * R + 2;  // sB row stride (doubles), the same
  static constexpr int kThreads = R == 4 ? 128 : 256, kCtas = 512 / kThreads;
  static constexpr int WC = R == 4 ? 1 : R / 8;  // column tiles per warp
  static constexpr int XS = kThreads / (KC * R);  // terms per sweep of the CTA
  // the term with recipe kCurlT (NX: none); its second operand is staged after the terms
  static constexpr int curl_term() {
    for (int x = 0; x < OP::NX; ++x)
      if (OP::recipe(x) == kCurlT) return x;
    return OP::NX;
  }
  static constexpr int kCurlX = curl_term();
  static constexpr bool kCurl = kCurlX < OP::NX;
  static constexpr int kA = OP::NT * KC * SA, kChunk = kA + (OP::NX + kCurl) * KC * SB;
  static constexpr int kRing = ring_depth(kChunk * 8, kCtas);
  static constexpr size_t smem = (size_t)kRing * kChunk * 8;
};

template <class OP, int R>
__global__ void __launch_bounds__(SynthCfg<OP, R>::kThreads, SynthCfg<OP, R>::kCtas)
    k_synth_f64(SynthArgs<OP::NX> a) {
  using C = SynthCfg<OP, R>;
  constexpr int NX = OP::NX, NP = OP::NP, NT = OP::NT, NO = OP::NO;
  constexpr int TH = C::TH, KC = C::KC, SA = C::SA, SB = C::SB, WC = C::WC;
  extern __shared__ __align__(16) double smem[];  // ring of [NT][KC][SA], [NX][KC][SB]

  const Tables& t = a.t;
  const int c0 = blockIdx.x * R;
  const int th0 = blockIdx.y * TH;
  const int mc = blockIdx.z;
  const int m = mc * t.minc;
  const int nlm = t.l_max - m + 1;
  const int ls = t.lstart[mc];
  const int nhs = t.nhs;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int rt = warp & 3, ctg = warp >> 2;

  const int nch = (nlm + KC - 1) / KC;
  auto chunk = [&](int c) { return smem + (c % C::kRing) * C::kChunk; };
  // this thread's row and column of the terms xb, xb + XS, ...
  const int xb = tid / (KC * R), kb = tid % (KC * R) / R, cb = tid % R;
  auto stage = [&](int c) {
    if (c < nch) {
      double* sA = chunk(c);
      double* sB = sA + C::kA;
      const int k0 = c * KC;
#pragma unroll
      for (int tb = 0; tb < NT; ++tb) {
        const double* T = (NT == 2) ? (tb == 0 ? t.plm : t.dplm)
                                    : (OP::table(0) == kP ? t.plm : t.dplm);
        stage_table<C::kThreads, KC, TH, SA>(sA + tb * KC * SA, T + (int64_t)ls * nhs, k0, nlm,
                                             th0, nhs);
      }
      const bool ok = k0 + kb < nlm && c0 + cb < a.ncols;
      const int64_t off = ok ? (int64_t)(ls + k0 + kb) * a.ld + c0 + cb : 0;
      double* d = sB + kb * SB + 2 * cb;
#pragma unroll
      for (int i = 0; i < (NX + C::XS - 1) / C::XS; ++i) {
        const int x = xb + C::XS * i;
        if (x < NX) cp16(d + x * KC * SB, a.src[x] + off, ok);
      }
      if (C::kCurl && xb == C::kCurlX % C::XS) cp16(d + NX * KC * SB, a.curl_b + off, ok);
    }
    cp_commit();
  };
  double or2[WC];
#pragma unroll
  for (int w = 0; w < WC; ++w) {
    const int col = c0 + 4 * (ctg * WC + w) + (g >> 1);
    or2[w] = C::kCurl && col < a.ncols ? __ldg(&a.or2[col]) : 0.0;
  }

  double acc[2][NP][WC][2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < NP; ++q)
#pragma unroll
      for (int w = 0; w < WC; ++w) acc[p][q][w][0] = acc[p][q][w][1] = 0.0;

#pragma unroll
  for (int c = 0; c < C::kRing - 1; ++c) stage(c);
  for (int c = 0; c < nch; ++c) {
    cp_wait<C::kRing - 2>();
    __syncthreads();  // chunk c is complete, and chunk c - 1's buffer free
    stage(c + C::kRing - 1);
    const double* sA = chunk(c);
    const double* sB = sA + C::kA;
#pragma unroll
    for (int par = 0; par < 2; ++par) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int kk = par + 2 * (4 * s + t4);
        const double l = (double)(m + c * KC + kk), dlh = l * (l + 1.0);
        double fa[NT];
#pragma unroll
        for (int tb = 0; tb < NT; ++tb) fa[tb] = sA[(tb * KC + kk) * SA + 8 * rt + g];
#pragma unroll
        for (int x = 0; x < NX; ++x) {  // one term at a time: fewer live registers
          double fb[WC];
#pragma unroll
          for (int w = 0; w < WC; ++w) {
            const double* b = &sB[(x * KC + kk) * SB + 8 * (ctg * WC + w) + g];
            fb[w] = *b;
            if (OP::recipe(x) == kDlh) fb[w] = dlh * fb[w];
            if (OP::recipe(x) == kCurlT) {
              const double f = or2[w] * dlh;
              fb[w] = f * fb[w] - b[(NX - x) * KC * SB];
            }
          }
#pragma unroll
          for (int q = 0; q < NP; ++q)
            if (OP::term(q) == x) {
              const int tb = (NT == 2) ? OP::table(q) : 0;
#pragma unroll
              for (int w = 0; w < WC; ++w) dmma(acc[par][q][w], fa[tb], fb[w]);
            }
        }
      }
    }
  }

  const int th = th0 + 8 * rt + g;
  if (th >= nhs) return;
  const double dm = (double)m;
#pragma unroll
  for (int w = 0; w < WC; ++w) {
    const int col = c0 + 4 * (ctg * WC + w) + t4;
    if (col >= a.ncols) continue;
    dcx hN[NP], hS[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      dcx E = {acc[0][q][w][0], acc[0][q][w][1]};
      dcx O = {acc[1][q][w][0], acc[1][q][w][1]};
      hN[q] = E + O;
      hS[q] = (OP::table(q) == kP) ? E - O : O - E;
    }
    dcx oN[NO], oS[NO];
    OP::combine(hN, dm, oN);
    OP::combine(hS, dm, oS);
    double2* FN = a.F + mc * a.f_m + (int64_t)(2 * th) * a.f_row + col * a.col_c;
    double2* FS = FN + a.f_row;
#pragma unroll
    for (int f = 0; f < NO; ++f) {
      FN[OP::field(f) * a.col_f] = make_double2(oN[f].x, oN[f].y);
      FS[OP::field(f) * a.col_f] = make_double2(oS[f].x, oS[f].y);
    }
  }
}

template <class OP, int R>
struct AnalCfg {
  static constexpr int TK = 64, KC = 16;
  static constexpr int SA = 18;         // sA row stride: rows 2 apart -> 32 B bank step
  static constexpr int SB = 2 * R + 4;  // sB row stride: 8*SB = 32 mod 128 B
  static constexpr int WC = R / 4;
  static constexpr int XS = 256 / (KC * R);  // fields per sweep of the CTA
  static constexpr int kSweeps = (OP::NX + XS - 1) / XS;
  static constexpr int kA = OP::NT * TK * SA, kChunk = kA + OP::NX * 2 * KC * SB;
  static constexpr int kRing = ring_depth(kChunk * 8);
  static constexpr size_t smem = (size_t)kRing * kChunk * 8;
};

template <class OP, int R>
__global__ void __launch_bounds__(256, 2) k_anal_f64(AnalArgs<OP::NX, OP::NO> a) {
  using C = AnalCfg<OP, R>;
  constexpr int NX = OP::NX, NP = OP::NP, NT = OP::NT, NO = OP::NO;
  constexpr int TK = C::TK, KC = C::KC, SA = C::SA, SB = C::SB, WC = C::WC;
  extern __shared__ __align__(16) double smem[];  // ring of [NT][TK][SA], [NX][2][KC][SB]

  const Tables& t = a.t;
  const int c0 = blockIdx.x * R;
  const int k0 = blockIdx.y * TK;
  const int mc = blockIdx.z;
  const int m = mc * t.minc;
  const int nlm = t.l_max - m + 1;
  if (k0 >= nlm) return;
  const int ls = t.lstart[mc];
  const int nhs = t.nhs;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int par = warp & 1;
  const int rowi = par + 2 * (8 * (warp >> 1) + g);  // row inside the 64-row tile

  const double2* Fm = a.F + mc * a.f_m;
  const int nch = (nhs + KC - 1) / KC;
  auto chunk = [&](int c) { return smem + (c % C::kRing) * C::kChunk; };
  // this thread's theta pair and column of the fields xb, xb + XS, ...: northern
  // row, and the southern one KC rows below
  const int xb = tid / (KC * R), jb = tid % (KC * R) / R, cb = tid % R;
  const int ob = xb * 2 * KC * SB + jb * SB + 2 * cb;
  auto stage = [&](int c) {
    if (c < nch) {
      double* sA = chunk(c);
      double* sB = sA + C::kA;
      const int j0 = c * KC;
#pragma unroll
      for (int tb = 0; tb < NT; ++tb)
        stage_table<256, TK, KC, SA>(sA + tb * TK * SA,
                                ((NT == 2 && tb) ? t.dplm : t.plm) + (int64_t)ls * nhs, k0, nlm,
                                j0, nhs);
      const bool ok = j0 + jb < nhs && c0 + cb < a.ncols;
      const double2* p =
          ok ? Fm + (int64_t)(2 * (j0 + jb)) * a.f_row + xb * a.col_x + (c0 + cb) * a.col_c : a.F;
#pragma unroll
      for (int i = 0; i < C::kSweeps; ++i)
        if (xb + C::XS * i < NX) {
          const double2* q = ok ? p + C::XS * i * a.col_x : p;
          cp16(sB + ob + C::XS * i * 2 * KC * SB, q, ok);
          cp16(sB + ob + (C::XS * i * 2 + 1) * KC * SB, ok ? q + a.f_row : q, ok);
        }
    }
    cp_commit();
  };
  // this thread's elements of chunk c: north and south rows -> sum and difference
  auto fold = [&](int c) {
    double* sB = chunk(c) + C::kA + ob;
#pragma unroll
    for (int i = 0; i < C::kSweeps; ++i)
      if (xb + C::XS * i < NX) {
        double2* n = reinterpret_cast<double2*>(sB + C::XS * i * 2 * KC * SB);
        double2* d = reinterpret_cast<double2*>(sB + (C::XS * i * 2 + 1) * KC * SB);
        const double2 vn = *n, vs = *d;
        *n = make_double2(vn.x + vs.x, vn.y + vs.y);
        *d = make_double2(vn.x - vs.x, vn.y - vs.y);
      }
  };

  double acc[NP][WC][2];
#pragma unroll
  for (int q = 0; q < NP; ++q)
#pragma unroll
    for (int w = 0; w < WC; ++w) acc[q][w][0] = acc[q][w][1] = 0.0;

#pragma unroll
  for (int c = 0; c < C::kRing - 1; ++c) stage(c);
  for (int c = 0; c < nch; ++c) {
    cp_wait<C::kRing - 2>();
    fold(c);
    __syncthreads();  // chunk c is complete, and chunk c - 1's buffer free
    stage(c + C::kRing - 1);
    const double* sA = chunk(c);
    const double* sB = sA + C::kA;
#pragma unroll
    for (int s = 0; s < KC / 4; ++s) {
      const int jj = 4 * s + t4;
      double fa[NT];
#pragma unroll
      for (int tb = 0; tb < NT; ++tb) fa[tb] = sA[(tb * TK + rowi) * SA + jj];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const int tb = (NT == 2) ? OP::table(q) : 0;
        // P rows: even -> north+south, odd -> north-south; dP the reverse
        const int sign = (OP::table(q) == kP) ? par : 1 - par;
        const double* b = &sB[((OP::term(q) * 2 + sign) * KC + jj) * SB + g];
#pragma unroll
        for (int w = 0; w < WC; ++w) dmma(acc[q][w], fa[tb], b[8 * w]);
      }
    }
  }

  // C fragment: row g of this warp's tile = k, complex column 4w + t4
  const int k = k0 + par + 2 * (8 * (warp >> 1) + g);
  if (k >= nlm) return;
  const double l = (double)(m + k);
  const double inv = (m + k) > 0 ? 1.0 / (l * (l + 1.0)) : 0.0;
  const double dm = (double)m;
#pragma unroll
  for (int w = 0; w < WC; ++w) {
    const int col = c0 + 4 * w + t4;
    if (col >= a.ncols) continue;
    dcx h[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) h[q] = {acc[q][w][0], acc[q][w][1]};
    dcx o[NO];
    OP::finish(h, dm, inv, o);
    const int64_t off = (int64_t)(ls + k) * a.ld + a.out_col0 + col;
#pragma unroll
    for (int f = 0; f < NO; ++f)
      if (a.out[f]) {
        a.out[f][off] = make_double2(o[f].x, o[f].y);
        if (a.zero_ends && col == 0) a.out[f][off - 1] = make_double2(0.0, 0.0);
        if (a.zero_ends && col == a.ncols - 1) a.out[f][off + 1] = make_double2(0.0, 0.0);
      }
  }
}

// ----------------------------------------------------------------- launchers

template <class OP, int R>
int launch_synth_f64(const SynthArgs<OP::NX>& a, cudaStream_t st) {
  using C = SynthCfg<OP, R>;
  static_assert(C::smem <= 113 * 1024, "synthesis ring too large");
  auto kern = k_synth_f64<OP, R>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)C::smem));
  dim3 grid((a.ncols + R - 1) / R, (a.t.nhs + C::TH - 1) / C::TH, a.t.n_m);
  kern<<<grid, C::kThreads, C::smem, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template <class OP, int R>
int launch_anal_f64(const AnalArgs<OP::NX, OP::NO>& a, cudaStream_t st) {
  using C = AnalCfg<OP, R>;
  static_assert(C::smem <= 113 * 1024, "analysis ring too large");
  auto kern = k_anal_f64<OP, R>;
  MT_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)C::smem));
  dim3 grid((a.ncols + R - 1) / R, (a.t.l_max + 1 + C::TK - 1) / C::TK, a.t.n_m);
  kern<<<grid, 256, C::smem, st>>>(a);
  MT_CHECK_CUDA(cudaGetLastError());
  return MT_OK;
}

template int launch_synth_f64<SynScalar, 16>(const SynthArgs<1>&, cudaStream_t);
template int launch_synth_f64<SynGrad<false>, 16>(const SynthArgs<1>&, cudaStream_t);
template int launch_synth_f64<SynGrad<true>, 16>(const SynthArgs<1>&, cudaStream_t);
template int launch_synth_f64<SynTorpol, 4>(const SynthArgs<3>&, cudaStream_t);
template int launch_synth_f64<SynGroups<2, 0>, 4>(const SynthArgs<6>&, cudaStream_t);
template int launch_synth_f64<SynGroups<2, 1>, 4>(const SynthArgs<7>&, cudaStream_t);
template int launch_synth_f64<SynGroups<2, 2>, 4>(const SynthArgs<8>&, cudaStream_t);
template int launch_synth_f64<SynAnelVel, 4>(const SynthArgs<4>&, cudaStream_t);
template int launch_synth_f64<SynAnelDr<1>, 4>(const SynthArgs<4>&, cudaStream_t);
template int launch_synth_f64<SynAnelDr<2>, 4>(const SynthArgs<5>&, cudaStream_t);
template int launch_anal_f64<AnaScalar, 8>(const AnalArgs<1, 1>&, cudaStream_t);
template int launch_anal_f64<AnaSphtor, 8>(const AnalArgs<2, 2>&, cudaStream_t);
template int launch_anal_f64<AnaGroups<1, 2>, 8>(const AnalArgs<6, 5>&, cudaStream_t);
template int launch_anal_f64<AnaGroups<1, 0>, 8>(const AnalArgs<3, 3>&, cudaStream_t);
template int launch_anal_f64<AnaGroups<2, 0>, 8>(const AnalArgs<3, 2>&, cudaStream_t);

}  // namespace mt
