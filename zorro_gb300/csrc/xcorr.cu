// Masked normalised cross-correlation windows (mnxc2, zorro.py:1014-1097).
//
// Every term of mnxc2 is real(IFFT_C(A * conj(B))) for two cropped spectra A
// and B of real images, and only the +/-maxShift window of it is ever used
// (zorro.py:1090-1092).  With the half-plane spectra of zr_spectra:
//
//   column pass  for each kx in [0, C1/2]: build the C0 products of column kx
//                exactly as the full C0 x C1 cropped product would contribute
//                to real(IFFT) (the Nyquist row/column of the crop is not its
//                own Hermitian mirror, so row ky=-C0/2 averages the -C0/2 and
//                +C0/2 products and column kx=C1/2 uses the mirrored -C1/2
//                values), inverse FFT of length C0, keep the w window rows;
//   row pass     two window rows packed into one complex inverse FFT of length
//                C1 (real-output trick), keep the w window columns, scale by
//                normConst2 (zorro.py:634; the inverse, like the reference's
//                FFTW execute(), carries no 1/N).
//
// The four frame-only terms (CorrTM, CorrBM and the two Denominator IFFTs)
// depend on one frame each, so they are computed once per frame (zr_xcorr_terms)
// instead of once per pair; the pair kernel only transforms the numerator
// G_J conj(G_I) and combines.  Since real(IFFT(A conj(B)))(y, x) =
// real(IFFT(conj(A) B))(-y, -x) for any spectra, CorrTM is CorrBM and DenomT
// is DenomB point-reflected: one transform per frame gives both, over the
// (w+1) x (w+1) window [-maxShift, maxShift]^2 that the reflection needs.
#include "common.cuh"
#include "fft_inplace.cuh"
#include "internal.h"

namespace zr {

// Column pass: columns per CTA (by default four, which write whole sectors of
// the window rows, and two from 2048 points on, where smaller CTAs overlap
// better: terms and 190 pair windows at crop 2048, 1193 us with four, 1143 us
// with two; at 1024, 608 and 615 us; the planner may choose 1, 2 or 4 per
// length).  Row pass: packed row pairs per CTA (default
// 2; the planner may choose 1, 2 or 4).
__host__ __device__ constexpr int xc_nbc_default(int C0) { return C0 >= 2048 ? 2 : 4; }
constexpr int XC_NBR_DEFAULT = 2;

struct XcJobs {
  const void* G;     // spectra: float2, or __half2 when ``sc`` is set
  const void* S;
  const void* GM;
  const int* pairs;  // kind 1
  const void* G2;    // kind 2: template spectra (triMode 'refine')
  const float* sc;   // half spectra: power-of-two scales, [N] G, [N] S, [1] GM
  int N;
  int kind;          // 0 terms, 1 pairs, 2 frame I against template I
  int job0;
  long long se;      // spectrum elements
  int rows;          // window rows kept by the column pass: w + 1 (terms) or w (pairs)
};

// The two spectra of a job (its product is A conj(B)) and, for half-precision
// spectra, the factor 1 / (scale_A scale_B) that undoes their scaling.
template <typename E>
__device__ __forceinline__ void job_operands(const XcJobs& J, int job, const E*& A, const E*& B, float& unscale) {
  const E* G = (const E*)J.G;
  int ia = 0, ib = 0;  // scale slots
  if (J.kind == 1) {
    const int I = J.pairs[2 * job], Jj = J.pairs[2 * job + 1];
    A = G + (size_t)Jj * J.se;
    B = G + (size_t)I * J.se;
    ia = Jj;
    ib = I;
  } else if (J.kind == 2) {  // base frame I, template (sum_n G_n - G_I) / N
    A = G + (size_t)job * J.se;
    B = (const E*)J.G2 + (size_t)job * J.se;
  } else {
    const int t = job / J.N, n = job - t * J.N;
    const E* GM = (const E*)J.GM;
    switch (t) {
      case 0: A = G + (size_t)n * J.se; B = GM; ia = n; break;                    // CorrBM (and CorrTM)
      case 1: A = (const E*)J.S + (size_t)n * J.se; B = GM; ia = J.N + n; break;  // DenomB (and DenomT)
      default: A = GM; B = GM; ia = 2 * J.N; break;                              // maskProduct
    }
    ib = 2 * J.N;
  }
  unscale = J.sc ? 1.0f / (J.sc[ia] * J.sc[ib]) : 1.0f;
}

// One complex value of a spectrum.
__device__ __forceinline__ float2 load_one(const float2* p) { return __ldg(p); }
__device__ __forceinline__ float2 load_one(const __half2* p) { return __half22float2(__ldg(p)); }
__device__ __forceinline__ float2 to_f2(float2 a) { return a; }
__device__ __forceinline__ float2 to_f2(__half2 a) { return __half22float2(a); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// Value of the cropped product A conj(B) at row ``row`` of column k, as the
// full C0 x C1 product contributes to real(IFFT): regular columns as they
// are, except that row C0/2 averages the -C0/2 and +C0/2 products (the
// latter stored at index C0 of the column); the Nyquist column C1/2 holds
// conj(A) B of the mirrored row; columns past it are zero.
template <int C0, typename E>
__device__ __forceinline__ float2 xc_product(const E* a, const E* b, int row, int k, int half, float us) {
  constexpr int hc = C0 / 2;
  float2 h = make_float2(0.0f, 0.0f);
  if (k < half) {
    h = cmulc(load_one(a + row), load_one(b + row));
    if (k > 0 && row == hc) {
      const float2 h2 = cmulc(load_one(a + C0), load_one(b + C0));
      h = make_float2(0.5f * (h.x + h2.x), 0.5f * (h.y + h2.y));
    }
  } else if (k == half) {
    const int m = row == 0 ? 0 : (row == hc ? C0 : C0 - row);
    h = cmulc(load_one(b + m), load_one(a + m));
  }
  if (sizeof(E) != sizeof(float2)) h = cscale(h, us);  // undo the power-of-two scales (exact)
  return h;
}

// Column pass: CTA (job, column group) transforms NBC columns of the
// job's product.  Jobs vary fastest across the grid, so the CTAs resident at
// one time read the same columns of every spectrum and share them through L2.
// The first FFT pass forms the products while it loads its butterflies from
// the (column-major) spectra.  The last pass computes the window rows
// [-maxShift, ...) alone: a window of at most NS rows takes at most one
// output of each RL-point butterfly, so it sums the twiddled inputs of those
// (PRUNED); a wider one (whole planes) runs the full butterflies.
template <int C0, typename E, int NBC, bool PRUNED>
__global__ void __launch_bounds__(ip_threads(C0, NBC), sm_minb(ip_threads(C0, NBC)))
    k_xc_cols(XcJobs J, int C1, int K4, int mS, float2* __restrict__ Tw, const float2* __restrict__ tw) {
  constexpr int T = ip_threads(C0, NBC);
  using P = Ip<C0>;
  constexpr int RP = C0 + 4;  // column pitch of the spectra
  extern __shared__ float2 sm[];
  const int k0 = blockIdx.y * NBC;
  const int jl = blockIdx.x;
  const E *A, *B;
  float us;
  job_operands(J, J.job0 + jl, A, B, us);
  const int half = C1 / 2;
  ip_pass1<C0, NBC, T, 1, false>(sm, [&](int b, int j, float2* v) {
    const int k = k0 + b;
    const E* a = A + (size_t)k * RP;
    const E* bb = B + (size_t)k * RP;
    if (k < half) {
      // every load of the butterfly first (all in bounds), then the products
      E av[16], bv[16];
#pragma unroll
      for (int r = 0; r < 16; r++) {
        av[r] = __ldg(a + j + r * P::A1);
        bv[r] = __ldg(bb + j + r * P::A1);
      }
#pragma unroll
      for (int r = 0; r < 16; r++) {
        float2 h = cmulc(to_f2(av[r]), to_f2(bv[r]));
        if (k > 0 && r == 8 && j == 0) {  // row -C0/2: average with the +C0/2 product
          const float2 h2 = cmulc(load_one(a + C0), load_one(bb + C0));
          h = make_float2(0.5f * (h.x + h2.x), 0.5f * (h.y + h2.y));
        }
        if (sizeof(E) != sizeof(float2)) h = cscale(h, us);  // undo the power-of-two scales (exact)
        v[r] = h;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 16; r++) v[r] = xc_product<C0>(a, bb, j + r * P::A1, k, half, us);
    }
  });
  __syncthreads();
  ip_pass2<C0, NBC, T, 1, false>(sm, tw);
  const int rows = J.rows;
  float2* out = Tw + (size_t)jl * rows * K4 + k0;
  if (PRUNED) {
    for (int e = threadIdx.x; e < rows * NBC; e += T) {
      const int a = e / NBC, c = e - a * NBC;
      out[(size_t)a * K4 + c] = ip_last_one<C0, NBC, 1>(sm, c, a - mS, tw);
    }
  } else {
    ip_last<C0, NBC, T, 1, true>(sm, tw, [&](int c, int k, const float2* v) {
#pragma unroll
      for (int r = 0; r < P::RL; r++) {  // y = k + r NS or that less C0 (both when 2 maxShift = C0)
        const int a0 = k + r * P::NS + mS, a1 = a0 - C0;
        if (a0 < rows) out[(size_t)a0 * K4 + c] = v[r];
        if (a1 >= 0) out[(size_t)a1 * K4 + c] = v[r];
      }
    });
  }
}

// Row pass: NBR pairs of window rows per CTA, each pair one complex inverse
// FFT; the last pass is pruned to the window columns like the column pass's.
template <int C1, int XC_NBR, bool PRUNED>
__global__ void __launch_bounds__(ip_threads(C1, XC_NBR), sm_minb(ip_threads(C1, XC_NBR)))
    k_xc_rows(XcJobs J, int C0, int K4, int mS, float scale, const float2* __restrict__ Tw,
              const float* __restrict__ terms, float* __restrict__ out, const float2* __restrict__ tw) {
  constexpr int T = ip_threads(C1, XC_NBR);
  using P = Ip<C1>;
  extern __shared__ float2 sm[];
  const int w = 2 * mS;
  const int rows = J.rows;  // w + 1 for the frame terms (rows and columns -mS..mS)
  const int jl = blockIdx.y;
  const int job = J.job0 + jl;
  const int arow0 = blockIdx.x * (2 * XC_NBR);
  // the pair's frames (read ahead of the transform)
  const int I = J.kind == 1 ? J.pairs[2 * job] : job, Jj = J.kind == 1 ? J.pairs[2 * job + 1] : job;
  const float2* src = Tw + (size_t)jl * rows * K4;
  ip_pass1<C1, XC_NBR, T, 1, false>(sm, [&](int p, int j, float2* v) {
    const int a0 = arow0 + 2 * p, a1 = a0 + 1;
    const float2* r0 = a0 < rows ? src + (size_t)a0 * K4 : nullptr;
    const float2* r1 = a1 < rows ? src + (size_t)a1 * K4 : nullptr;
#pragma unroll
    for (int r = 0; r < 16; r++) v[r] = packed_rows<C1>(r0, r1, j + r * P::A1);
  });
  __syncthreads();
  ip_pass2<C1, XC_NBR, T, 1, false>(sm, tw);
  const size_t w2 = (size_t)w * w;
  const int cols = rows;  // the terms window is square, w + 1 wide
  // Window element (a, b) of a frame term; elements (a, b) and (a + 1, b) of a
  // pair, whose ten term values are all loaded before either is combined (one
  // row after the other, the frame numbers read beside them: 190 windows and
  // terms at crop 2048 1145 us, 1129 so; 66 windows at crop 128 24.2 and 23.0)
  auto emit_terms = [&](int a, int b, float v) {
    if (a >= rows) return;
    v *= scale;
    const size_t pix = (size_t)a * w + b;
    // output slots: CorrTM [0,N), CorrBM [N,2N), DenomT [2N,3N), DenomB [3N,4N), maskProduct 4N
    const int t = job / J.N, n = job - t * J.N;
    const int main_slot = t == 0 ? J.N + n : (t == 1 ? 3 * J.N + n : 4 * J.N);
    if (a < w && b < w) out[(size_t)main_slot * w2 + pix] = v;
    if (t < 2 && a >= 1 && b >= 1) {
      const int refl_slot = t == 0 ? n : 2 * J.N + n;
      out[(size_t)refl_slot * w2 + (size_t)(w - a) * w + (w - b)] = v;
    }
  };
  auto emit_pair = [&](int a, int b, float2 v) {
    const int N = J.N;
    const float* base[5] = {terms + (size_t)I * w2, terms + (size_t)(N + Jj) * w2, terms + (size_t)(2 * N + I) * w2,
                            terms + (size_t)(3 * N + Jj) * w2, terms + (size_t)(4 * N) * w2};
    const size_t pix = (size_t)a * w + b;
    float t[2][5];  // every load before any value is used
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
      for (int i = 0; i < 5; i++) t[q][i] = a + q < rows ? base[i][pix + q * w] : 1.0f;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const float ctm = t[q][0], cbm = t[q][1], dt = t[q][2], db = t[q][3], mp = t[q][4];
      float den = sqrtf((db - cbm * (cbm / mp)) * (dt - ctm * (ctm / mp)));
      den = (den < 1.0f) ? 1.0f : den;  // np.clip(Denom, 1, inf); NaN stays NaN
      if (a + q < rows) out[(size_t)job * w2 + pix + q * w] = ((q == 0 ? v.x : v.y) * scale - ctm * cbm / mp) / den;
    }
  };
  if (!PRUNED) {
    ip_last_inplace<C1, XC_NBR, T, 1>(sm, tw);
    __syncthreads();
  }
  for (int e = threadIdx.x; e < XC_NBR * cols; e += T) {
    const int p = e / cols, b = e - p * cols;
    const int x = b - mS;
    const float2 v = PRUNED ? ip_last_one<C1, XC_NBR, 1>(sm, p, x, tw)
                            : sm[p * ip_ld(C1, XC_NBR) + ip_at<C1>(x < 0 ? x + C1 : x)];
    if (J.kind == 0) {
      emit_terms(arow0 + 2 * p, b, v.x);
      emit_terms(arow0 + 2 * p + 1, b, v.y);
    } else {
      emit_pair(arow0 + 2 * p, b, v);
    }
  }
}

template <int C0, typename E, int NBC, bool PRUNED>
static int launch_xc_cols_t(const XcJobs& J, int nj, int C1, int K4, int mS, float2* Tw, const float2* tw,
                            cudaStream_t st) {
  constexpr int T = ip_threads(C0, NBC);
  const size_t smem = (size_t)NBC * ip_ld(C0, NBC) * sizeof(float2);
  const auto kern = k_xc_cols<C0, E, NBC, PRUNED>;
  ZR_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_xc_cols attr"));
  kern<<<dim3(nj, K4 / NBC), T, smem, st>>>(J, C1, K4, mS, Tw, tw);
  return launched("k_xc_cols");
}

template <int C0, typename E, bool PRUNED>
static int launch_xc_cols_e(const XcJobs& J, int nj, int C1, int K4, int mS, float2* Tw, const float2* tw,
                            cudaStream_t st) {
  switch (tune_get(TUNE_XC_COLS, C0)) {
    case 1: return launch_xc_cols_t<C0, E, 1, PRUNED>(J, nj, C1, K4, mS, Tw, tw, st);
    case 2: return launch_xc_cols_t<C0, E, 2, PRUNED>(J, nj, C1, K4, mS, Tw, tw, st);
    case 4: return launch_xc_cols_t<C0, E, 4, PRUNED>(J, nj, C1, K4, mS, Tw, tw, st);
    default: return launch_xc_cols_t<C0, E, xc_nbc_default(C0), PRUNED>(J, nj, C1, K4, mS, Tw, tw, st);
  }
}

template <int C0>
static int launch_xc_cols(const XcJobs& J, int nj, int C1, int K4, int mS, float2* Tw, const float2* tw,
                          cudaStream_t st) {
  const bool pruned = J.rows <= Ip<C0>::NS;
  if (J.sc)
    return pruned ? launch_xc_cols_e<C0, __half2, true>(J, nj, C1, K4, mS, Tw, tw, st)
                  : launch_xc_cols_e<C0, __half2, false>(J, nj, C1, K4, mS, Tw, tw, st);
  return pruned ? launch_xc_cols_e<C0, float2, true>(J, nj, C1, K4, mS, Tw, tw, st)
                : launch_xc_cols_e<C0, float2, false>(J, nj, C1, K4, mS, Tw, tw, st);
}

template <int C1, int NBR, bool PRUNED>
static int launch_xc_rows_v(const XcJobs& J, int nj, int C0, int K4, int mS, float scale, const float2* Tw,
                            const float* terms, float* out, const float2* tw, cudaStream_t st) {
  constexpr int T = ip_threads(C1, NBR);
  const size_t smem = (size_t)NBR * ip_ld(C1, NBR) * sizeof(float2);
  const auto kern = k_xc_rows<C1, NBR, PRUNED>;
  ZR_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_xc_rows attr"));
  kern<<<dim3((J.rows + 2 * NBR - 1) / (2 * NBR), nj), T, smem, st>>>(J, C0, K4, mS, scale, Tw, terms, out, tw);
  return launched("k_xc_rows");
}

template <int C1, bool PRUNED>
static int launch_xc_rows_p(const XcJobs& J, int nj, int C0, int K4, int mS, float scale, const float2* Tw,
                            const float* terms, float* out, const float2* tw, cudaStream_t st) {
  switch (tune_get(TUNE_XC_ROWS, C1)) {
    case 1: return launch_xc_rows_v<C1, 1, PRUNED>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st);
    case 2: return launch_xc_rows_v<C1, 2, PRUNED>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st);
    case 4: return launch_xc_rows_v<C1, 4, PRUNED>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st);
    default: return launch_xc_rows_v<C1, XC_NBR_DEFAULT, PRUNED>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st);
  }
}

template <int C1>
static int launch_xc_rows(const XcJobs& J, int nj, int C0, int K4, int mS, float scale, const float2* Tw,
                          const float* terms, float* out, const float2* tw, cudaStream_t st) {
  return J.rows <= Ip<C1>::NS ? launch_xc_rows_p<C1, true>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st)
                              : launch_xc_rows_p<C1, false>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st);
}

#define ZR_XC_DISPATCH(L, CALL)                               \
  switch (L) {                                                \
    case 64: { constexpr int LL = 64; CALL; } break;          \
    case 128: { constexpr int LL = 128; CALL; } break;        \
    case 256: { constexpr int LL = 256; CALL; } break;        \
    case 512: { constexpr int LL = 512; CALL; } break;        \
    case 384: { constexpr int LL = 384; CALL; } break;        \
    case 768: { constexpr int LL = 768; CALL; } break;        \
    case 1024: { constexpr int LL = 1024; CALL; } break;      \
    case 1536: { constexpr int LL = 1536; CALL; } break;      \
    case 2048: { constexpr int LL = 2048; CALL; } break;      \
    case 3072: { constexpr int LL = 3072; CALL; } break;      \
    case 4096: { constexpr int LL = 4096; CALL; } break;      \
    default: return set_error(ZR_ESIZE, "crop size %d not supported", (int)(L)); \
  }

static int run_jobs(XcJobs J, int njobs, int C0, int C1, int mS, const float* terms, float* out, void* work,
                    size_t work_bytes, cudaStream_t st) {
  const int K4 = zr_spectrum_pitch(C1);
  const size_t per_job = (size_t)J.rows * K4 * sizeof(float2);
  if (!work || work_bytes < per_job)
    return set_error(ZR_EWORK, "zr_xcorr: work buffer %zu bytes < %zu (one job)", work_bytes, per_job);
  const int wave = (int)((work_bytes / per_job) < (size_t)njobs ? work_bytes / per_job : (size_t)njobs);
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  // normConst2 (zorro.py:634, rounded to float32 as there); the reference's
  // inverse FFTs are FFTW executions without 1/N, and so is this one
  const float scale = (float)(1.0 / (((double)C0 * C1) * ((double)C0 * C1)));
  float2* Tw = (float2*)work;
  for (int j0 = 0; j0 < njobs; j0 += wave) {
    const int nj = (njobs - j0) < wave ? (njobs - j0) : wave;
    J.job0 = j0;
    ZR_XC_DISPATCH(C0, ZR_TRY((launch_xc_cols<LL>(J, nj, C1, K4, mS, Tw, tw, st))));
    ZR_XC_DISPATCH(C1, ZR_TRY((launch_xc_rows<LL>(J, nj, C0, K4, mS, scale, Tw, terms, out, tw, st))));
  }
  return ZR_OK;
}

static int check_sizes(int C0, int C1, int mS) {
  if (!fft_len_ok(C0) || !fft_len_ok(C1) || C0 < 64 || C1 < 64 || C0 > 4096 || C1 > 4096)
    return set_error(ZR_ESIZE, "crop %dx%d must be powers of two in [64, 4096] or 3 x 2^k in [384, 3072]", C0, C1);
  if (mS < 2 || 2 * mS > C0 || 2 * mS > C1)
    return set_error(ZR_ESIZE, "maxShift %d must satisfy 2 <= maxShift <= C/2", mS);
  return ZR_OK;
}

// triMode 'refine' (zorro.py:934-954): template I is conj(sum_n G_n - G_I)/N.
// One thread per spectrum element: the frame sum in frame order, then every
// frame's template.
__global__ void k_refine_spectra(const float2* __restrict__ G, int N, long long se, float2* __restrict__ T) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= se) return;
  float sx = 0.0f, sy = 0.0f;
  for (int n = 0; n < N; n++) {
    const float2 g = G[(size_t)n * se + e];
    sx += g.x;
    sy += g.y;
  }
  const float fn = (float)N;
  for (int n = 0; n < N; n++) {
    const float2 g = G[(size_t)n * se + e];
    T[(size_t)n * se + e] = make_float2((sx - g.x) / fn, (sy - g.y) / fn);
  }
}

// The template's frame terms are linear in its spectra: CorrTM and the raw
// DenomT of template I are (sum_n term_n - term_I) / N.  CorrBM, DenomB and
// the mask product are copied.
__global__ void k_refine_terms(const float* __restrict__ terms, int N, int w2, float* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= w2) return;
  const float fn = (float)N;
  for (int t = 0; t < 4; t += 2) {  // CorrTM (slots [0,N)) and DenomT (slots [2N,3N))
    const float* src = terms + (size_t)t * N * w2;
    float s = 0.0f;
    for (int n = 0; n < N; n++) s += src[(size_t)n * w2 + p];
    for (int n = 0; n < N; n++) out[((size_t)t * N + n) * w2 + p] = (s - src[(size_t)n * w2 + p]) / fn;
  }
  for (int n = 0; n < N; n++) {
    out[((size_t)N + n) * w2 + p] = terms[((size_t)N + n) * w2 + p];
    out[((size_t)3 * N + n) * w2 + p] = terms[((size_t)3 * N + n) * w2 + p];
  }
  out[(size_t)4 * N * w2 + p] = terms[(size_t)4 * N * w2 + p];
}

// Half-precision spectra: each spectrum is stored as __half2 times a power of
// two chosen from its largest component, max * scale < 2^15.
__global__ void k_spectrum_absmax(const float2* __restrict__ X, long long se, unsigned int* __restrict__ maxbits) {
  const float2* x = X + (size_t)blockIdx.y * se;
  float m = 0.0f;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < se; e += (long long)gridDim.x * blockDim.x) {
    const float2 v = x[e];
    m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits + blockIdx.y, __float_as_uint(m));  // m >= 0: bits order as values
}

__device__ __forceinline__ float half_scale(unsigned int bits) {
  const float m = __uint_as_float(bits);
  if (!(m > 0.0f) || isinf(m)) return 1.0f;
  int ex;
  frexpf(m, &ex);  // m < 2^ex
  return ldexpf(1.0f, 15 - ex);
}

__global__ void k_spectrum_to_half(const float2* __restrict__ X, long long se, const unsigned int* __restrict__ maxbits,
                                   __half2* __restrict__ Y, float* __restrict__ scales) {
  const int n = blockIdx.y;
  const float sc = half_scale(maxbits[n]);
  if (blockIdx.x == 0 && threadIdx.x == 0) scales[n] = sc;
  const float2* x = X + (size_t)n * se;
  __half2* y = Y + (size_t)n * se;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < se; e += (long long)gridDim.x * blockDim.x) {
    const float2 v = x[e];
    y[e] = __floats2half2_rn(v.x * sc, v.y * sc);
  }
}

}  // namespace zr

using namespace zr;

extern "C" int zr_pack_half(const void* spectra, int n_spectra, long long se, void* out, float* scales, void* work,
                            size_t work_bytes, void* stream) {
  if (!spectra || !out || !scales || !work || n_spectra <= 0 || se <= 0)
    return set_error(ZR_EINVAL, "zr_pack_half: bad argument");
  if (work_bytes < (size_t)n_spectra * sizeof(unsigned int))
    return set_error(ZR_EWORK, "zr_pack_half: work buffer %zu < %zu", work_bytes, (size_t)n_spectra * 4);
  cudaStream_t st = (cudaStream_t)stream;
  ZR_TRY(cuda_check(cudaMemsetAsync(work, 0, (size_t)n_spectra * sizeof(unsigned int), st), "zr_pack_half memset"));
  const int blocks = (int)((se + 255) / 256 < 304 ? (se + 255) / 256 : 304);
  k_spectrum_absmax<<<dim3(blocks, n_spectra), 256, 0, st>>>((const float2*)spectra, se, (unsigned int*)work);
  ZR_TRY(launched("k_spectrum_absmax"));
  k_spectrum_to_half<<<dim3(blocks, n_spectra), 256, 0, st>>>((const float2*)spectra, se, (const unsigned int*)work,
                                                               (__half2*)out, scales);
  return launched("k_spectrum_to_half");
}

extern "C" int zr_refine_spectra(const void* G, int N, int C0, int C1, void* templates, void* stream) {
  if (!G || !templates || N <= 0) return set_error(ZR_EINVAL, "zr_refine_spectra: null argument");
  const long long se = zr_spectrum_elems(C0, C1);
  k_refine_spectra<<<(unsigned)((se + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const float2*)G, N, se,
                                                                                    (float2*)templates);
  return launched("k_refine_spectra");
}

extern "C" int zr_refine_terms(const float* terms, int N, int max_shift, float* out, void* stream) {
  if (!terms || !out || N <= 0 || max_shift <= 0) return set_error(ZR_EINVAL, "zr_refine_terms: bad argument");
  const int w2 = 4 * max_shift * max_shift;
  k_refine_terms<<<(w2 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(terms, N, w2, out);
  return launched("k_refine_terms");
}

extern "C" int zr_xcorr_refine(const void* G, const void* templates, const float* refine_terms, int N, int C0,
                               int C1, int max_shift, float* cwin, void* work, size_t work_bytes, void* stream) {
  if (!G || !templates || !refine_terms || !cwin || N <= 0) return set_error(ZR_EINVAL, "zr_xcorr_refine: null argument");
  if (N < 2) return ZR_OK;
  ZR_TRY(check_sizes(C0, C1, max_shift));
  XcJobs J{G, nullptr, nullptr, nullptr, templates, nullptr, N, 2, 0, zr_spectrum_elems(C0, C1), 2 * max_shift};
  return run_jobs(J, N - 1, C0, C1, max_shift, refine_terms, cwin, work, work_bytes, (cudaStream_t)stream);
}

extern "C" size_t zr_xcorr_work_bytes(int n_jobs, int C1, int max_shift) {
  return (size_t)n_jobs * (2 * max_shift + 1) * zr_spectrum_pitch(C1) * sizeof(float2);
}

extern "C" int zr_xcorr_terms(const void* G, const void* S, const void* GM, int N, int C0, int C1, int max_shift,
                              float* terms, void* work, size_t work_bytes, void* stream) {
  if (!G || !S || !GM || !terms || N <= 0) return set_error(ZR_EINVAL, "zr_xcorr_terms: null argument");
  ZR_TRY(check_sizes(C0, C1, max_shift));
  XcJobs J{G, S, GM, nullptr, nullptr, nullptr, N, 0, 0, zr_spectrum_elems(C0, C1), 2 * max_shift + 1};
  return run_jobs(J, 2 * N + 1, C0, C1, max_shift, nullptr, terms, work, work_bytes, (cudaStream_t)stream);
}

extern "C" int zr_xcorr_pairs(const void* G, const float* terms, const int* pairs, int M, int N, int C0, int C1,
                              int max_shift, float* cwin, void* work, size_t work_bytes, void* stream) {
  if (!G || !terms || !pairs || !cwin || N <= 0) return set_error(ZR_EINVAL, "zr_xcorr_pairs: null argument");
  if (M <= 0) return ZR_OK;
  ZR_TRY(check_sizes(C0, C1, max_shift));
  XcJobs J{G, nullptr, nullptr, pairs, nullptr, nullptr, N, 1, 0, zr_spectrum_elems(C0, C1), 2 * max_shift};
  return run_jobs(J, M, C0, C1, max_shift, terms, cwin, work, work_bytes, (cudaStream_t)stream);
}

extern "C" int zr_xcorr_terms_half(const void* G, const void* S, const void* GM, const float* scales, int N, int C0,
                                   int C1, int max_shift, float* terms, void* work, size_t work_bytes, void* stream) {
  if (!G || !S || !GM || !scales || !terms || N <= 0) return set_error(ZR_EINVAL, "zr_xcorr_terms_half: null argument");
  ZR_TRY(check_sizes(C0, C1, max_shift));
  XcJobs J{G, S, GM, nullptr, nullptr, scales, N, 0, 0, zr_spectrum_elems(C0, C1), 2 * max_shift + 1};
  return run_jobs(J, 2 * N + 1, C0, C1, max_shift, nullptr, terms, work, work_bytes, (cudaStream_t)stream);
}

extern "C" int zr_xcorr_pairs_half(const void* G, const float* scales, const float* terms, const int* pairs, int M,
                                   int N, int C0, int C1, int max_shift, float* cwin, void* work, size_t work_bytes,
                                   void* stream) {
  if (!G || !scales || !terms || !pairs || !cwin || N <= 0) return set_error(ZR_EINVAL, "zr_xcorr_pairs_half: null argument");
  if (M <= 0) return ZR_OK;
  ZR_TRY(check_sizes(C0, C1, max_shift));
  XcJobs J{G, nullptr, nullptr, pairs, nullptr, scales, N, 1, 0, zr_spectrum_elems(C0, C1), 2 * max_shift};
  return run_jobs(J, M, C0, C1, max_shift, terms, cwin, work, work_bytes, (cudaStream_t)stream);
}
