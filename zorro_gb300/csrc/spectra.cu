// Forward spectra of the masked frames (xcorrnm2_tri, zorro.py:814-925).
//
// The reference transforms m*I and (m*I)^2 as two complex P0 x P1 FFTs per
// frame and keeps the four corners (FFTCrop, zorro.py:901-914).  Here both
// real images go through ONE complex FFT per row (z = u + i u^2, untangled by
// Hermitian symmetry), only the C1/2+1 non-negative kx columns the crop keeps
// are written, and the column pass keeps only the C0+1 cropped ky rows.
//
// Row-pass output layout (scratch): [frame][y/8][K4][y%8] complex (the last
// group of a frame as many rows as it has, a multiple of 4): the row pass's
// stores of consecutive k lie close together, and two columns of 8 rows are
// the 128-byte line that eight and eight lanes of the column pass read.
#include <stdio.h>

#include <type_traits>

#include "common.cuh"
#include "fft_inplace.cuh"
#include "internal.h"

namespace zr {

constexpr int NBR = 8;  // rows per group of the row-pass output layout
// Element (k, y) of one frame's row-pass output of 4 H4 rows.
__device__ __forceinline__ int ru_rows(int y, int H4) { return min(NBR, 4 * H4 - (y & ~(NBR - 1))); }
__device__ __forceinline__ size_t ru_at(int k, int y, int K4, int H4) {
  return (size_t)(y & ~(NBR - 1)) * K4 + (size_t)k * ru_rows(y, H4) + (y & (NBR - 1));
}
// Rows per CTA of the row pass and columns per CTA of the column pass: the
// defaults, or the planner's choice of 1, 2 or 4 per transform length
// (tune_get).  Two rows of 4096 points make two CTAs an SM, of which one loads
// while the other transforms.  Spectra of eight K2 frames, microseconds, with
// R rows and C columns a CTA and groups of G rows: 634 with R 4, C 1, G 16;
// 639 with R 2, C 1, G 16; 630 with R 4, C 2, G 8; 589 with R 2, C 2, G 8; 595
// with R 2, C 2, G 4; 780 with R 1 (8-byte stores).  Below 2048 points several
// CTAs of four rows share an SM anyway: eight frames of 1000 x 1000, 43.6 with
// R 2, 39.9 with R 4; of 2000 x 2000, 151 and 152.
constexpr int FC_DEFAULT = 2;
__host__ __device__ constexpr int fr_default(int P1) { return P1 >= 2048 ? 2 : 4; }
// CTAs per SM to ask the register allocator for: 128 registers a thread
constexpr int minb_of(int T) { return sm_minb(T); }

// corrected16 for x and x + 1 (x = j + r STEP, j even): u0 holds pixels x +
// odd, u1 x + 1 - odd.  Needs even row lengths and frame strides and arrays
// aligned to two elements (wide_pixels).  Half the loads of corrected16, which
// waited for them: spectra of eight K2 frames 671 -> 645 us.
template <int STEP, int FULL>
__device__ __forceinline__ void corrected32(const FrameSrc& f, int n, int y, int j, int cols, int odd, float* u0,
                                            float* u1) {
  const int lim = cols - j;
  const long long q = (long long)y * f.W + j;
  const long long p = q + map_off(f, n);
  const long long i = (long long)n * f.fstride + q;
#define ZR_INSIDE(r) (r < FULL || r * STEP < lim)
  float2 u[16];
  if (f.type == ZR_U8) {
    unsigned short bits[16];
#pragma unroll
    for (int r = 0; r < 16; r++)
      bits[r] = ZR_INSIDE(r) ? __ldg((const unsigned short*)((const uint8_t*)f.raw + i + r * STEP)) : 0;
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = make_float2((float)(bits[r] & 255), (float)(bits[r] >> 8));
  } else if (f.type == ZR_F32) {
#pragma unroll
    for (int r = 0; r < 16; r++)
      u[r] = ZR_INSIDE(r) ? __ldg((const float2*)((const float*)f.raw + i + r * STEP)) : make_float2(0.0f, 0.0f);
  } else {
    unsigned int bits[16];
#pragma unroll
    for (int r = 0; r < 16; r++)
      bits[r] = ZR_INSIDE(r) ? __ldg((const unsigned int*)((const uint16_t*)f.raw + i + r * STEP)) : 0u;
#pragma unroll
    for (int r = 0; r < 16; r++) {
      if (f.type == ZR_F16)
        u[r] = make_float2(__half2float(__ushort_as_half((unsigned short)(bits[r] & 0xffffu))),
                           __half2float(__ushort_as_half((unsigned short)(bits[r] >> 16))));
      else u[r] = make_float2((float)(bits[r] & 0xffffu), (float)(bits[r] >> 16));
    }
  }
  auto map = [&](const float* m, int r) {
    return ZR_INSIDE(r) ? __ldg((const float2*)(m + p + r * STEP)) : make_float2(0.0f, 0.0f);
  };
  if (f.gain) {
    float2 g[16];
#pragma unroll
    for (int r = 0; r < 16; r++) g[r] = map(f.gain, r);
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = make_float2(__fmul_rn(g[r].x, u[r].x), __fmul_rn(g[r].y, u[r].y));
  }
  if (f.gdiv != 0.0f) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = make_float2(__fdiv_rn(u[r].x, f.gdiv), __fdiv_rn(u[r].y, f.gdiv));
  }
  if (f.ha) {
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      float2 a[8], b[8];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        a[r] = map(f.ha, h + r);
        b[r] = map(f.hb, h + r);
      }
#pragma unroll
      for (int r = 0; r < 8; r++)
        u[h + r] = make_float2(__fmaf_rn(a[r].x, u[h + r].x, b[r].x), __fmaf_rn(a[r].y, u[h + r].y, b[r].y));
    }
  }
#undef ZR_INSIDE
#pragma unroll
  for (int r = 0; r < 16; r++) {
    u0[r] = odd ? u[r].y : u[r].x;
    u1[r] = odd ? u[r].x : u[r].y;
  }
}

// Row pass: FR rows of one frame per CTA.  The first FFT pass reads the
// pixels (consecutive lanes, consecutive pixels) and the last one untangles
// the half-plane rows of u and u^2 in registers, so the rows pass through
// shared memory twice and the CTA meets at two barriers.  MASKS: frames under a
// mask, and masks themselves (a kernel of their own: in one with the plain
// frames their loads made those spill, spectra of eight K2 frames 588 -> 596 us).
template <int P1, int FR, bool MASKS>
__global__ void __launch_bounds__(ip_threads(P1, FR), minb_of(ip_threads(P1, FR)))
    k_fwd_rows(FrameSrc f, const float* __restrict__ mask, const double* __restrict__ mean_sub,
               double inv_area, int frame0, int mode, int rows, int cols, int C1, int K4, int H4, bool wide,
               float2* __restrict__ RU, float2* __restrict__ RV, const float2* __restrict__ tw) {
  constexpr int T = ip_threads(P1, FR);
  using P = Ip<P1>;
  extern __shared__ float2 sm[];
  // frames vary fastest so that concurrent CTAs read the same rows of the
  // gain and hot-pixel maps through L2
  const int y0 = blockIdx.y * FR;
  const int nl = blockIdx.x;
  const int n = frame0 + nl;
  float mu = 0.0f;
  if ((!MASKS || mode == 0) && mean_sub) mu = (float)(mean_sub[n] * inv_area);
  if constexpr (MASKS) {
    if (mode == 0) {
      ip_pass1<P1, FR, T, -1, false>(sm, [&](int b, int j, float2* v) {
        const int y = y0 + b, lim = y < rows ? cols - j : 0;
        const float* m = mask + (size_t)y * P1 + j;
        float u[16], k[16];
#pragma unroll
        for (int r = 0; r < 16; r++) k[r] = r * P::A1 < lim ? __ldg(m + r * P::A1) : 0.0f;
        if (y < rows) corrected16<P::A1, 0>(f, n, y, j, cols, u);
#pragma unroll
        for (int r = 0; r < 16; r++) {
          const float w = r * P::A1 < lim ? k[r] * (u[r] - mu) : 0.0f;
          v[r] = make_float2(w, w * w);
        }
      });
    } else if (mask) {  // the mask itself
      ip_pass1<P1, FR, T, -1, false>(sm, [&](int b, int j, float2* v) {
        const int y = y0 + b, lim = y < rows ? cols - j : 0;
        const float* m = mask + (size_t)y * P1 + j;
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = make_float2(r * P::A1 < lim ? __ldg(m + r * P::A1) : 0.0f, 0.0f);
      });
    } else {  // (ones inside the frame)
      ip_pass1<P1, FR, T, -1, false>(sm, [&](int b, int j, float2* v) {
        const int lim = y0 + b < rows ? cols - j : 0;
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = make_float2(r * P::A1 < lim ? 1.0f : 0.0f, 0.0f);
      });
    }
  } else if (wide) {
    auto pixels = [&](auto full) {
      constexpr int FULL = decltype(full)::value;
      ip_pass1_pairs<P1, FR, T, -1>(sm, [&](int b, int j, int odd, float2* v0, float2* v1) {
        const int y = y0 + b;
        if (y >= rows) {
#pragma unroll
          for (int r = 0; r < 16; r++) v0[r] = v1[r] = make_float2(0.0f, 0.0f);
          return;
        }
        float u0[16], u1[16];
        corrected32<P::A1, FULL>(f, n, y, j, cols, odd, u0, u1);
        const int lim = cols - j;
#pragma unroll
        for (int r = 0; r < 16; r++) {
          const bool in = r < FULL || r * P::A1 < lim;
          const float a = in ? u0[r] - mu : 0.0f, b = in ? u1[r] - mu : 0.0f;
          v0[r] = make_float2(a, a * a);
          v1[r] = make_float2(b, b * b);
        }
      });
    };
    if (cols >= 14 * P::A1) pixels(std::integral_constant<int, 14>());
    else pixels(std::integral_constant<int, 0>());
  } else {
    auto pixels = [&](auto full) {
      constexpr int FULL = decltype(full)::value;
      ip_pass1<P1, FR, T, -1, false>(sm, [&](int b, int j, float2* v) {
        const int y = y0 + b;
        if (y >= rows) {
#pragma unroll
          for (int r = 0; r < 16; r++) v[r] = make_float2(0.0f, 0.0f);
          return;
        }
        float u[16];
        corrected16<P::A1, FULL>(f, n, y, j, cols, u);
        const int lim = cols - j;
#pragma unroll
        for (int r = 0; r < 16; r++) {
          const float w = r < FULL || r * P::A1 < lim ? u[r] - mu : 0.0f;
          v[r] = make_float2(w, w * w);
        }
      });
    };
    // pixels that need no test against the row's end (frames fill most of
    // their padded rows)
    if (cols >= 14 * P::A1) pixels(std::integral_constant<int, 14>());
    else pixels(std::integral_constant<int, 0>());
  }
  __syncthreads();
  ip_pass2<P1, FR, T, -1, false>(sm, tw);
  const int half = C1 / 2;
  const size_t frame_out = (size_t)nl * 4 * H4 * K4;
  const int step = ru_rows(y0, H4);  // between consecutive k (the CTA's rows share a group)
  ip_last_paired<P1, FR, T, -1>(sm, tw, [&](int b, int k0, const float2* X0, int k1, const float2* X1) {
    if ((y0 + b) >> 2 >= H4) return;
    const size_t o = frame_out + ru_at(0, y0 + b, K4, H4);
    float2 *ou = RU + o, *ov = RV + o;
    auto put = [&](int k, float2 zk, float2 zm) {
      ou[k * step] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
      if (!MASKS || mode == 0) ov[k * step] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    };
#pragma unroll
    for (int q = 0; q < P::RL; q++) {
      const int m0 = k0 + q * P::NS, m1 = k1 + q * P::NS;
      if (m0 <= half) put(m0, X0[q], k0 > 0 ? X1[P::RL - 1 - q] : X0[(P::RL - q) % P::RL]);
      if (m1 <= half) put(m1, X1[q], k0 > 0 ? X0[P::RL - 1 - q] : X1[P::RL - 1 - q]);
    }
  });
  // the pitch's columns past C1/2 are zero
  for (int e = threadIdx.x; e < FR * (K4 - half - 1); e += T) {
    const int b = e % FR, k = half + 1 + e / FR;
    if ((y0 + b) >> 2 >= H4) continue;
    const size_t o = frame_out + ru_at(k, y0 + b, K4, H4);
    RU[o] = make_float2(0.0f, 0.0f);
    if (!MASKS || mode == 0) RV[o] = make_float2(0.0f, 0.0f);
  }
}

// Column pass: FC columns of one spectrum per CTA, read from the row pass's
// output by the first FFT pass (zero past the frame: the zero padding to P0)
// and written by the last one: consecutive lanes hold consecutive ky.
template <int P0, int FC>
__global__ void __launch_bounds__(ip_threads(P0, FC), minb_of(ip_threads(P0, FC)))
    k_fwd_cols(const float2* __restrict__ RU, const float2* __restrict__ RV, int rows, int C0, int K4, int H4,
               long long spec_elems, float2* __restrict__ G, float2* __restrict__ S,
               const float2* __restrict__ tw) {
  constexpr int T = ip_threads(P0, FC);
  using P = Ip<P0>;
  extern __shared__ float2 sm[];
  const int k0 = blockIdx.x * FC;
  const int nl = blockIdx.y;
  const float2* R = (blockIdx.z == 0 ? RU : RV) + (size_t)nl * 4 * H4 * K4;
  const int hc = C0 / 2;
  const int RP = C0 + 4;
  float2* out = (blockIdx.z == 0 ? G : S) + (size_t)nl * spec_elems + (size_t)k0 * RP;
  // (whole groups of rows and a butterfly step of whole groups: one stride)
  const bool even = H4 % (NBR / 4) == 0 && P::A1 % NBR == 0;
  ip_pass1<P0, FC, T, -1, true>(sm, [&](int c, int j, float2* v) {
    if (even) {
      const float2* src = R + (size_t)(j & ~(NBR - 1)) * K4 + (k0 + c) * NBR + (j & (NBR - 1));
      const size_t step = (size_t)P::A1 * K4;
      const int lim = rows - j;
#pragma unroll
      for (int r = 0; r < 16; r++) {
        v[r] = make_float2(0.0f, 0.0f);
        if (r * P::A1 < lim) v[r] = __ldg(src);
        src += step;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 16; r++) {
        const int y = j + r * P::A1;
        v[r] = y < rows ? __ldg(R + ru_at(k0 + c, y, K4, H4)) : make_float2(0.0f, 0.0f);
      }
    }
  });
  // rows C0 + 1 .. C0 + 3 pad the column to its pitch: written as zeros, so
  // that every element of a spectrum is defined (zr_pack_half scans them all)
  for (int e = threadIdx.x; e < 3 * FC; e += T) out[(size_t)(e / 3) * RP + C0 + 1 + e % 3] = make_float2(0.0f, 0.0f);
  __syncthreads();
  ip_pass2<P0, FC, T, -1, false>(sm, tw);
  ip_last<P0, FC, T, -1, false>(sm, tw, [&](int c, int k, const float2* v) {
    float2* col = out + (size_t)c * RP;
#pragma unroll
    for (int r = 0; r < P::RL; r++) {
      const int ky = k + r * P::NS;
      if (ky < hc) col[ky] = v[r];
      if (ky == hc) col[C0] = v[r];
      if (ky >= P0 - hc) col[ky - (P0 - C0)] = v[r];
    }
  });
}

__global__ void k_frame_sums(FrameSrc f, double* __restrict__ sums) {
  const int n = blockIdx.y;
  const long long npix = (long long)f.H * f.W;
  float acc = 0.0f;
  double dacc = 0.0;
  int cnt = 0;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npix;
       p += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(p / f.W), x = (int)(p - (long long)y * f.W);
    acc += load_corrected(f, n, y, x);
    if (++cnt == 64) { dacc += acc; acc = 0.0f; cnt = 0; }
  }
  dacc += acc;
  for (int o = 16; o > 0; o >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dacc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) atomicAdd(sums + n, v);
  }
}

// Frames whose pixels can be read two at a time.
static bool wide_pixels(const FrameSrc& f, int cols) {
  const int esize = f.type == ZR_U8 ? 1 : (f.type == ZR_F32 ? 4 : 2);
  const uintptr_t maps = (uintptr_t)f.gain | (uintptr_t)f.ha | (uintptr_t)f.hb;
  return (f.W & 1) == 0 && (cols & 1) == 0 && (f.fstride & 1) == 0 && (f.mstride & 1) == 0 && (maps & 7) == 0 &&
         (uintptr_t)f.raw % (2 * esize) == 0;
}

template <int P, int FR, bool MASKS>
static int launch_rows_m(const FrameSrc& f, const float* mask, const double* mean_sub, double inv_area,
                         int frame0, int nfr, int mode, int rows, int cols, int C1, int K4, int H4,
                         float2* RU, float2* RV, const float2* tw, cudaStream_t st) {
  constexpr int T = ip_threads(P, FR);
  const size_t smem = (size_t)FR * ip_ld(P, FR) * sizeof(float2);
  ZR_TRY(cuda_check(cudaFuncSetAttribute(k_fwd_rows<P, FR, MASKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_fwd_rows attr"));
  k_fwd_rows<P, FR, MASKS><<<dim3(nfr, (rows + FR - 1) / FR), T, smem, st>>>(f, mask, mean_sub, inv_area, frame0, mode,
                                                                              rows, cols, C1, K4, H4,
                                                                              wide_pixels(f, cols), RU, RV, tw);
  return launched("k_fwd_rows");
}

template <int P, int FR>
static int launch_rows_v(const FrameSrc& f, const float* mask, const double* mean_sub, double inv_area,
                         int frame0, int nfr, int mode, int rows, int cols, int C1, int K4, int H4,
                         float2* RU, float2* RV, const float2* tw, cudaStream_t st) {
  const auto run = mask || mode != 0 ? launch_rows_m<P, FR, true> : launch_rows_m<P, FR, false>;
  return run(f, mask, mean_sub, inv_area, frame0, nfr, mode, rows, cols, C1, K4, H4, RU, RV, tw, st);
}

template <int P>
static int launch_rows(const FrameSrc& f, const float* mask, const double* mean_sub, double inv_area,
                       int frame0, int nfr, int mode, int rows, int cols, int C1, int K4, int H4,
                       float2* RU, float2* RV, const float2* tw, cudaStream_t st) {
  switch (tune_get(TUNE_FWD_ROWS, P)) {
    case 1: return launch_rows_v<P, 1>(f, mask, mean_sub, inv_area, frame0, nfr, mode, rows, cols, C1, K4, H4, RU, RV, tw, st);
    case 2: return launch_rows_v<P, 2>(f, mask, mean_sub, inv_area, frame0, nfr, mode, rows, cols, C1, K4, H4, RU, RV, tw, st);
    case 4: return launch_rows_v<P, 4>(f, mask, mean_sub, inv_area, frame0, nfr, mode, rows, cols, C1, K4, H4, RU, RV, tw, st);
    default:
      return launch_rows_v<P, fr_default(P)>(f, mask, mean_sub, inv_area, frame0, nfr, mode, rows, cols, C1, K4, H4, RU, RV,
                                          tw, st);
  }
}

template <int P, int FC>
static int launch_cols_v(const float2* RU, const float2* RV, int rows, int C0, int K4, int H4, long long se,
                         int nfr, int nz, float2* G, float2* S, const float2* tw, cudaStream_t st) {
  constexpr int T = ip_threads(P, FC);
  const size_t smem = (size_t)FC * ip_ld(P, FC) * sizeof(float2);
  ZR_TRY(cuda_check(cudaFuncSetAttribute(k_fwd_cols<P, FC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_fwd_cols attr"));
  k_fwd_cols<P, FC><<<dim3(K4 / FC, nfr, nz), T, smem, st>>>(RU, RV, rows, C0, K4, H4, se, G, S, tw);
  return launched("k_fwd_cols");
}

template <int P>
static int launch_cols(const float2* RU, const float2* RV, int rows, int C0, int K4, int H4, long long se,
                       int nfr, int nz, float2* G, float2* S, const float2* tw, cudaStream_t st) {
  switch (tune_get(TUNE_FWD_COLS, P)) {
    case 1: return launch_cols_v<P, 1>(RU, RV, rows, C0, K4, H4, se, nfr, nz, G, S, tw, st);
    case 2: return launch_cols_v<P, 2>(RU, RV, rows, C0, K4, H4, se, nfr, nz, G, S, tw, st);
    case 4: return launch_cols_v<P, 4>(RU, RV, rows, C0, K4, H4, se, nfr, nz, G, S, tw, st);
    default: return launch_cols_v<P, FC_DEFAULT>(RU, RV, rows, C0, K4, H4, se, nfr, nz, G, S, tw, st);
  }
}

#define ZR_POW2_DISPATCH(L, CALL)                  \
  switch (L) {                                     \
    case 64: { constexpr int LL = 64; CALL; } break;     \
    case 128: { constexpr int LL = 128; CALL; } break;   \
    case 256: { constexpr int LL = 256; CALL; } break;   \
    case 512: { constexpr int LL = 512; CALL; } break;   \
    case 1024: { constexpr int LL = 1024; CALL; } break; \
    case 1536: { constexpr int LL = 1536; CALL; } break; \
    case 2048: { constexpr int LL = 2048; CALL; } break; \
    case 3072: { constexpr int LL = 3072; CALL; } break; \
    case 4096: { constexpr int LL = 4096; CALL; } break; \
    case 6144: { constexpr int LL = 6144; CALL; } break; \
    default: return set_error(ZR_ESIZE, "transform length %d not supported (powers of two 64..4096, 1536, 3072, 6144)", (int)(L)); \
  }

}  // namespace zr

using namespace zr;

extern "C" int zr_spectrum_pitch(int C1) { return ((C1 / 2 + 1) + 3) & ~3; }

extern "C" long long zr_spectrum_elems(int C0, int C1) { return (long long)(C0 + 4) * zr_spectrum_pitch(C1); }

extern "C" size_t zr_spectra_work_bytes(int height, int n_frames, int C1) {
  const size_t H4 = (size_t)(height + 3) / 4;
  return 2 * (size_t)n_frames * H4 * zr_spectrum_pitch(C1) * 4 * sizeof(float2);
}

extern "C" int zr_frame_sums(const zr_frames_t* frames, double* sums, void* stream) {
  if (!frames || !sums || !frames->raw) return set_error(ZR_EINVAL, "zr_frame_sums: null argument");
  FrameSrc f = make_src(frames);
  if (f.N <= 0 || f.H <= 0 || f.W <= 0) return set_error(ZR_EINVAL, "zr_frame_sums: empty movie");
  const long long npix = (long long)f.H * f.W;
  int bx = (int)((npix + 256 * 64 - 1) / (256 * 64));
  if (bx > 1024) bx = 1024;
  k_frame_sums<<<dim3(bx, f.N), 256, 0, (cudaStream_t)stream>>>(f, sums);
  return launched("k_frame_sums");
}

extern "C" int zr_spectra(const zr_frames_t* frames, const float* mask, const double* mean_sub, int frame0,
                          int n_frames, int mode, int P0, int P1, int C0, int C1, void* G, void* S, void* work,
                          size_t work_bytes, void* stream) {
  if (!frames || !G || (mode == 0 && (!S || !frames->raw)))
    return set_error(ZR_EINVAL, "zr_spectra: null argument");
  if (!fft_len_ok(P0) || !fft_len_ok(P1) || !fft_len_ok(C0) || !fft_len_ok(C1) || C0 > P0 || C1 > P1 || C0 < 64 ||
      C1 < 64 || P0 > 6144 || P1 > 6144 || C0 > 4096 || C1 > 4096)
    return set_error(ZR_ESIZE,
                     "zr_spectra: P=%dx%d C=%dx%d must be powers of two or 3 x 2^k with 64 <= C <= P, P <= 6144, "
                     "C <= 4096", P0, P1, C0, C1);
  FrameSrc f = make_src(frames);
  if (f.H > P0 || f.W > P1) return set_error(ZR_EINVAL, "zr_spectra: frame %dx%d larger than padded %dx%d", f.H, f.W, P0, P1);
  if (n_frames <= 0 || frame0 < 0 || (mode == 0 && frame0 + n_frames > f.N))
    return set_error(ZR_EINVAL, "zr_spectra: frame range [%d,%d) outside movie of %d frames", frame0, frame0 + n_frames, f.N);
  const int rows = (mode == 1 && mask) ? P0 : f.H;
  const int cols = (mode == 1 && mask) ? P1 : f.W;
  const int H4 = (rows + 3) / 4;
  const int K4 = zr_spectrum_pitch(C1);
  const size_t need = (size_t)(mode == 0 ? 2 : 1) * n_frames * H4 * K4 * 4 * sizeof(float2);
  if (!work || work_bytes < need)
    return set_error(ZR_EWORK, "zr_spectra: work buffer %zu bytes < %zu needed", work_bytes, need);
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  float2* RU = (float2*)work;
  float2* RV = RU + (size_t)n_frames * H4 * K4 * 4;
  cudaStream_t st = (cudaStream_t)stream;
  const double inv_area = 1.0 / ((double)f.H * f.W);
  ZR_POW2_DISPATCH(P1, ZR_TRY((launch_rows<LL>(f, mask, mean_sub, inv_area, frame0, n_frames, mode, rows, cols, C1,
                                                K4, H4, RU, RV, tw, st))));
  const long long se = zr_spectrum_elems(C0, C1);
  ZR_POW2_DISPATCH(P0, ZR_TRY((launch_cols<LL>(RU, RV, rows, C0, K4, H4, se, n_frames, mode == 0 ? 2 : 1,
                                                (float2*)G, (float2*)S, tw, st))));
  return ZR_OK;
}
