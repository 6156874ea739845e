// Dose-weighted sum (doseFilter, zorro.py:2349-2494), the Unblur filter:
//
//   filtSum = | IFFT( sum_n FFT(pad_sym(frame_n)) * thres_n(q) * filt_n(q) ) |[:H, :W]
//   filt_n(q)  = exp(-0.5 * dose_end_n / critDose(q)),
//   critDose(q) = vs * (A q^B + C)   (the value at the Nyquist corner is
//                 replaced by the square of its left neighbour, zorro.py:2422),
//   thres_n(q) = exp(-(q / thresQ_n)^order).
//
// The filters are real and even in frequency, so the accumulated spectrum is
// Hermitian: only kx in [0, P1/2] is kept.  Two aligned frames share one
// complex row FFT; the column pass applies each frame's filter and
// accumulates in registers; the inverse column pass keeps only the H output
// rows and the final row pass packs two rows per complex inverse FFT.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "fft_inplace.cuh"
#include "internal.h"

namespace zr {

// rows per CTA of the forward row pass, columns per CTA of the inverse column
// pass
__host__ __device__ constexpr int ds_rows(int P1) { return P1 >= 3072 ? 2 : 4; }
constexpr int DS_NBR = 4;
constexpr int DS_G = 8;  // rows per group of the row pass's output

// Element (k, y) of one frame's row-pass output.
__device__ __forceinline__ size_t rw_at(int k, int y, int K4) {
  return ((size_t)(y / DS_G) * K4 + k) * DS_G + y % DS_G;
}
// columns per CTA for a transform of length L: two for the 6144-point
// transforms, whose four-column tiles would not fit the register file
__host__ __device__ constexpr int ds_nbr(int L) { return L > 4096 ? 2 : DS_NBR; }
// CTAs per SM to ask the register allocator for: 128 registers a thread
constexpr int ds_minb(int T) { return sm_minb(T); }

__device__ __forceinline__ int sym_idx(int i, int n) {
  int m = i % (2 * n);
  return m < n ? m : 2 * n - 1 - m;
}

// Forward row pass: two or four rows of two frames per CTA, one complex
// transform a row.  What bounds it: the latency of its loads and the scattered
// stores (issue slots 35 % and shared-memory bandwidth 48 % used).  So a thread
// loads two columns at a time, several CTAs share an SM (two of two rows from
// 3072 points on), and a row's stores lie within DS_G rows of one another (as
// columns of the whole height every 32 bytes went to a line 32 KB from the
// last).  40 K2 frames, the whole filter: 2395 us with four rows a CTA, single
// columns and whole columns; 2235 us so; 2330 us with four rows, 2359 us with
// groups of four.  At 2048 points four rows take 324 us for 20 frames of 2000 x
// 2000, two rows 364 us; at 1024, 93 us for 1000 x 1000 and 101 us.
template <int P1>
__global__ void __launch_bounds__(ip_threads(P1, ds_rows(P1)), ds_minb(ip_threads(P1, ds_rows(P1))))
    k_dose_rows(const float* __restrict__ img, int N, int H, int W, int f0, int K4, int P0, bool wide,
                float2* __restrict__ RW, const float2* __restrict__ tw) {
  constexpr int NB = ds_rows(P1);
  constexpr int T = ip_threads(P1, NB);
  using P = Ip<P1>;
  extern __shared__ float2 sm[];
  const int y0 = blockIdx.x * NB;
  const int pl = blockIdx.y;              // frame pair within the chunk
  const int na = f0 + 2 * pl, nb = na + 1;
  const float* ia = img + (size_t)na * H * W;
  const float* ib = img + (size_t)(nb < N ? nb : na) * H * W;
  // row b: the symmetric padding of the two frames' row
  auto source = [&](int b) {
    const int yy = y0 + b;
    return (size_t)(yy < H ? yy : (yy < 2 * H ? 2 * H - 1 - yy : sym_idx(yy, H))) * W;
  };
  auto column = [&](int x) { return x < W ? x : (x < 2 * W ? 2 * W - 1 - x : sym_idx(x, W)); };
  if (wide && W >= 14 * P::A1) {  // two columns a load
    ip_pass1_pairs<P1, NB, T, -1>(sm, [&](int b, int j, int odd, float2* v0, float2* v1) {
      const size_t row = source(b);
      const float *pa = ia + row, *pb = ib + row;
      float2 a[16], c[16];
#pragma unroll
      for (int r = 0; r < 16; r++) {
        const int x = j + r * P::A1;
        if (r < 14 || x < W) {
          a[r] = __ldg(reinterpret_cast<const float2*>(pa + x));
          c[r] = nb < N ? __ldg(reinterpret_cast<const float2*>(pb + x)) : make_float2(0.0f, 0.0f);
        } else {
          const int x0 = column(x), x1 = column(x + 1);
          a[r] = make_float2(__ldg(pa + x0), __ldg(pa + x1));
          c[r] = nb < N ? make_float2(__ldg(pb + x0), __ldg(pb + x1)) : make_float2(0.0f, 0.0f);
        }
      }
#pragma unroll
      for (int r = 0; r < 16; r++) {
        v0[r] = odd ? make_float2(a[r].y, c[r].y) : make_float2(a[r].x, c[r].x);
        v1[r] = odd ? make_float2(a[r].x, c[r].x) : make_float2(a[r].y, c[r].y);
      }
    });
  } else {
    ip_pass1<P1, NB, T, -1, false>(sm, [&](int b, int j, float2* v) {
      const size_t row = source(b);
      const float *pa = ia + row, *pb = ib + row;
#pragma unroll
      for (int r = 0; r < 16; r++) {
        const int xs = column(j + r * P::A1);
        v[r] = make_float2(__ldg(pa + xs), nb < N ? __ldg(pb + xs) : 0.0f);
      }
    });
  }
  __syncthreads();
  ip_pass2<P1, NB, T, -1, false>(sm, tw);
  // output: [frame][ky / DS_G][kx][ky % DS_G]; the last pass pairs X[k] with
  // X[P1 - k] in registers
  const size_t fa = (size_t)(2 * pl) * K4 * P0;
  const size_t fb = fa + (size_t)K4 * P0;
  ip_last_paired<P1, NB, T, -1>(sm, tw, [&](int r, int k0, const float2* x0, int k1, const float2* x1) {
    auto put = [&](int k, float2 zk, float2 zm) {
      const size_t o = rw_at(k, y0 + r, K4);
      RW[fa + o] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
      if (nb < N) RW[fb + o] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    };
#pragma unroll
    for (int q = 0; q < P::RL; q++) {
      const int m0 = k0 + q * P::NS, m1 = k1 + q * P::NS;
      if (m0 <= P1 / 2) put(m0, x0[q], k0 > 0 ? x1[P::RL - 1 - q] : x0[(P::RL - q) % P::RL]);
      if (m1 <= P1 / 2) put(m1, x1[q], k0 > 0 ? x0[P::RL - 1 - q] : x1[P::RL - 1 - q]);
    }
  });
  // the pitch's columns past P1/2 are zero
  for (int e = threadIdx.x; e < NB * (K4 - P1 / 2 - 1); e += T) {
    const int r = e % NB, k = P1 / 2 + 1 + e / NB;
    const size_t o = rw_at(k, y0 + r, K4);
    RW[fa + o] = make_float2(0.0f, 0.0f);
    if (nb < N) RW[fb + o] = make_float2(0.0f, 0.0f);
  }
}

__device__ __forceinline__ float crit_dose(const zr_dose_params_t& p, int fy, int fx) {
  const float q = sqrtf((float)fx * (float)fx * (p.inv_ps_x * p.inv_ps_x) + (float)fy * (float)fy * (p.inv_ps_y * p.inv_ps_y));
  return p.voltage_scaling * (p.crit_a * powf(q, p.crit_b) + p.crit_c);
}

// The whole filter of 40 K2 frames went from 2708 to 2395 us with the in-place
// transforms (fft_inplace.cuh) and to 2235 us with the row pass above; the row
// and column passes' intermediates (2.7 GB each way) and the 2.3 GB of frames
// take 1130 us of it at copy bandwidth.
//
// One column kx per CTA: for every frame, the column's forward FFT, times the
// frame's filter, accumulated in registers: thread k holds the rows k + r NS
// that its last-pass butterfly puts out, so the spectrum is weighted and
// summed straight from that pass.
__host__ __device__ constexpr int ds_ct(int P0) { return P0 / ip_rl(P0) < 64 ? 64 : P0 / ip_rl(P0); }

template <int P0>
__global__ void __launch_bounds__(ds_ct(P0), ds_minb(ds_ct(P0)))
    k_dose_cols(const float2* __restrict__ RW, int f0, int nfr, int K4, int P1, zr_dose_params_t prm,
                const float* __restrict__ thres_q, const float* __restrict__ dose_end, int first,
                float2* __restrict__ ACC, float* __restrict__ FM, const float2* __restrict__ tw) {
  constexpr int T = ds_ct(P0);
  using P = Ip<P0>;
  extern __shared__ float2 sm[];
  // per-element constants of this column: 1/critDose(q) and log2(q)
  float* inv_crit = reinterpret_cast<float*>(sm + ip_ld(P0, 1));
  float* lq = inv_crit + P0;
  const int kx = blockIdx.x;
  const bool live = kx <= P1 / 2;
  for (int y = threadIdx.x; y < P0 && live; y += T) {
    const int fy = y < P0 / 2 ? y : y - P0;
    const float q = sqrtf((float)kx * (float)kx * (prm.inv_ps_x * prm.inv_ps_x) +
                          (float)fy * (float)fy * (prm.inv_ps_y * prm.inv_ps_y));
    float crit;
    if (y == P0 / 2 && kx == P1 / 2) {
      const float c = crit_dose(prm, fy, P1 / 2 - 1);
      crit = c * c;  // zorro.py:2422
    } else {
      crit = prm.voltage_scaling * (prm.crit_a * powf(q, prm.crit_b) + prm.crit_c);
    }
    inv_crit[y] = 1.0f / crit;
    lq[y] = log2f(q);
  }
  // (256 points: 16 butterflies of 16 outputs, shared by 64 threads through
  // shared memory)
  constexpr bool SPREAD = P::NS < T;
  constexpr int PER = SPREAD ? P0 / T : P::RL, STEP = SPREAD ? T : P::NS;
  static_assert(STEP == T, "every thread holds its rows");
  float2 acc[PER];
  float fm[PER];
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const size_t o = (size_t)kx * P0 + threadIdx.x + r * STEP;
    acc[r] = first ? make_float2(0.0f, 0.0f) : ACC[o];
    fm[r] = (first || !prm.normalize) ? 0.0f : FM[o];
  }
  const float LOG2E = 1.4426950408889634f;
  for (int nl = 0; nl < nfr; nl++) {
    const float2* col = RW + (size_t)nl * K4 * P0;
    // filt = exp(-0.5 D / crit), thres = exp(-(q / thresQ)^order)
    const float cd = (-0.5f * dose_end[f0 + nl]) * LOG2E;
    const float ltq = log2f(thres_q[f0 + nl]);
    __syncthreads();  // the previous frame's spectrum has been read
    ip_pass1<P0, 1, T, -1, false>(sm, [&](int, int j, float2* v) {
#pragma unroll
      for (int r = 0; r < 16; r++) v[r] = __ldg(col + rw_at(kx, j, K4) + (size_t)r * P::A1 * K4);
    });
    __syncthreads();
    ip_pass2<P0, 1, T, -1, false>(sm, tw);
    if (SPREAD) {
      ip_last_inplace<P0, 1, T, -1>(sm, tw);
      __syncthreads();
    }
    if (live) {
      float2 v[PER];
      if constexpr (SPREAD) {
#pragma unroll
        for (int r = 0; r < PER; r++) v[r] = sm[ip_at<P0>(threadIdx.x + r * STEP)];
      } else {
        ip_last_load<P0, 1>(sm, 0, threadIdx.x, v);
        ip_twiddle_last<P0, -1>(v, threadIdx.x, tw);
        ip_dft<P::RL, -1>(v);
      }
#pragma unroll
      for (int r = 0; r < PER; r++) {
        const int y = threadIdx.x + r * STEP;
        const float filt = exp2f(cd * inv_crit[y]);
        const float thres = exp2f(-LOG2E * exp2f(prm.cutoff_order * (lq[y] - ltq)));
        const float w = thres * filt;
        acc[r] = make_float2(acc[r].x + v[r].x * w, acc[r].y + v[r].y * w);
        if (prm.normalize) fm[r] += w;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < PER; r++) {
    const size_t o = (size_t)kx * P0 + threadIdx.x + r * STEP;
    ACC[o] = acc[r];
    if (prm.normalize) FM[o] = fm[r];
  }
}

// Inverse column pass, keeping rows [0, H).
template <int P0>
__global__ void __launch_bounds__(ip_threads(P0, ds_nbr(P0)), ds_minb(ip_threads(P0, ds_nbr(P0))))
    k_dose_icols(const float2* __restrict__ ACC, const float* __restrict__ FM, int normalize, int K4, int H,
                 float2* __restrict__ T2, const float2* __restrict__ tw) {
  constexpr int NB = ds_nbr(P0);
  constexpr int T = ip_threads(P0, NB);
  using P = Ip<P0>;
  extern __shared__ float2 sm[];
  const int k0 = blockIdx.x * NB;
  ip_pass1<P0, NB, T, 1, false>(sm, [&](int c, int j, float2* v) {
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const size_t o = (size_t)(k0 + c) * P0 + j + r * P::A1;
      v[r] = __ldg(ACC + o);
      if (normalize) {
        const float s = 1.0f / (__ldg(FM + o) + 1.0f);
        v[r] = make_float2(v[r].x * s, v[r].y * s);
      }
    }
  });
  __syncthreads();
  ip_pass2<P0, NB, T, 1, false>(sm, tw);
  ip_last<P0, NB, T, 1, true>(sm, tw, [&](int c, int k, const float2* v) {
#pragma unroll
    for (int r = 0; r < P::RL; r++) {
      const int y = k + r * P::NS;
      if (y < H) T2[(size_t)y * K4 + k0 + c] = v[r];
    }
  });
}

// Real-output inverse row pass (two rows per complex FFT), |.|, crop, scale.
template <int P1>
__global__ void __launch_bounds__(ip_threads(P1, 2), ds_minb(ip_threads(P1, 2)))
    k_dose_irows(const float2* __restrict__ T2, int K4, int H, int W, float scale, float* __restrict__ out,
                 const float2* __restrict__ tw) {
  constexpr int T = ip_threads(P1, 2);
  using P = Ip<P1>;
  extern __shared__ float2 sm[];
  const int y0 = blockIdx.x * 4;
  ip_pass1<P1, 2, T, 1, false>(sm, [&](int p, int j, float2* v) {
    const int a0 = y0 + 2 * p, a1 = a0 + 1;
    const float2* r0 = a0 < H ? T2 + (size_t)a0 * K4 : nullptr;
    const float2* r1 = a1 < H ? T2 + (size_t)a1 * K4 : nullptr;
#pragma unroll
    for (int r = 0; r < 16; r++) v[r] = packed_rows<P1>(r0, r1, j + r * P::A1);
  });
  __syncthreads();
  ip_pass2<P1, 2, T, 1, false>(sm, tw);
  ip_last<P1, 2, T, 1, false>(sm, tw, [&](int p, int k, const float2* v) {
    const int y = y0 + 2 * p;
    float* o = out + (size_t)y * W;
#pragma unroll
    for (int r = 0; r < P::RL; r++) {
      const int x = k + r * P::NS;
      if (x >= W) continue;
      if (y < H) o[x] = fabsf(v[r].x * scale);
      if (y + 1 < H) o[W + x] = fabsf(v[r].y * scale);
    }
  });
}

template <int P>
static int set_smem(const void* fn, size_t smem) {
  return cuda_check(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "dose attr");
}

#define ZR_DOSE_DISPATCH(L, CALL)                               \
  switch (L) {                                                  \
    case 256: { constexpr int LL = 256; CALL; } break;          \
    case 512: { constexpr int LL = 512; CALL; } break;          \
    case 1024: { constexpr int LL = 1024; CALL; } break;        \
    case 1536: { constexpr int LL = 1536; CALL; } break;        \
    case 2048: { constexpr int LL = 2048; CALL; } break;        \
    case 3072: { constexpr int LL = 3072; CALL; } break;        \
    case 4096: { constexpr int LL = 4096; CALL; } break;        \
    case 6144: { constexpr int LL = 6144; CALL; } break;        \
    default: return set_error(ZR_ESIZE, "dose filter size %d not supported", (int)(L)); \
  }

template <int P1>
static int dose_rows(const float* img, int N, int H, int W, int f0, int npairs, int K4, int P0, float2* RW,
                     const float2* tw, cudaStream_t st) {
  constexpr int T = ip_threads(P1, ds_rows(P1));
  const size_t smem = (size_t)ds_rows(P1) * ip_ld(P1, ds_rows(P1)) * sizeof(float2);
  const bool wide = (W & 1) == 0 && ((uintptr_t)img & 7) == 0;  // every row starts on 8 bytes
  ZR_TRY(set_smem<P1>((const void*)k_dose_rows<P1>, smem));
  k_dose_rows<P1><<<dim3(P0 / ds_rows(P1), npairs), T, smem, st>>>(img, N, H, W, f0, K4, P0, wide, RW, tw);
  return launched("k_dose_rows");
}

template <int P0>
static int dose_cols(const float2* RW, int f0, int nfr, int K4, int P1, const zr_dose_params_t& prm,
                     const float* tq, const float* de, int first, float2* ACC, float* FM, const float2* tw,
                     cudaStream_t st) {
  const size_t smem = (size_t)ip_ld(P0, 1) * sizeof(float2) + (size_t)2 * P0 * sizeof(float);
  ZR_TRY(set_smem<P0>((const void*)k_dose_cols<P0>, smem));
  k_dose_cols<P0><<<K4, ds_ct(P0), smem, st>>>(RW, f0, nfr, K4, P1, prm, tq, de, first, ACC, FM, tw);
  return launched("k_dose_cols");
}

template <int P0>
static int dose_icols(const float2* ACC, const float* FM, int normalize, int K4, int H, float2* T2, const float2* tw,
                      cudaStream_t st) {
  const size_t smem = (size_t)ds_nbr(P0) * ip_ld(P0, ds_nbr(P0)) * sizeof(float2);
  ZR_TRY(set_smem<P0>((const void*)k_dose_icols<P0>, smem));
  k_dose_icols<P0><<<K4 / ds_nbr(P0), ip_threads(P0, ds_nbr(P0)), smem, st>>>(ACC, FM, normalize, K4, H, T2, tw);
  return launched("k_dose_icols");
}

template <int P1>
static int dose_irows(const float2* T2, int K4, int H, int W, float scale, float* out, const float2* tw,
                      cudaStream_t st) {
  const size_t smem = (size_t)2 * ip_ld(P1, 2) * sizeof(float2);
  ZR_TRY(set_smem<P1>((const void*)k_dose_irows<P1>, smem));
  k_dose_irows<P1><<<(H + 3) / 4, ip_threads(P1, 2), smem, st>>>(T2, K4, H, W, scale, out, tw);
  return launched("k_dose_irows");
}

}  // namespace zr

using namespace zr;

static size_t dose_fixed_bytes(int P0, int P1) {
  const size_t K4 = zr_spectrum_pitch(P1);
  return (size_t)P0 * K4 * (2 * sizeof(float2) + sizeof(float));
}

static size_t dose_frame_bytes(int P0, int P1) { return (size_t)P0 * zr_spectrum_pitch(P1) * sizeof(float2); }

extern "C" size_t zr_dose_work_bytes(int P0, int P1, int n_frames) {
  return dose_fixed_bytes(P0, P1) + (size_t)n_frames * dose_frame_bytes(P0, P1);
}

extern "C" int zr_dose_filter(const float* aligned, int N, int H, int W, const zr_dose_params_t* params,
                              const float* thres_q, const float* dose_end, int P0, int P1, float* filt_sum,
                              void* work, size_t work_bytes, void* stream) {
  if (!aligned || !params || !thres_q || !dose_end || !filt_sum || !work)
    return set_error(ZR_EINVAL, "zr_dose_filter: null argument");
  if (N <= 0 || H <= 0 || W <= 0 || H > P0 || W > P1) return set_error(ZR_EINVAL, "zr_dose_filter: bad sizes");
  if (!fft_len_ok(P0) || !fft_len_ok(P1) || P0 < 256 || P1 < 256 || P0 > 6144 || P1 > 6144 || P0 == 8192 ||
      P1 == 8192)
    return set_error(ZR_ESIZE,
                     "zr_dose_filter: padded size %dx%d must be a power of two in [256, 4096], 1536, 3072 or 6144", P0,
                     P1);
  const size_t fixed = dose_fixed_bytes(P0, P1), per = dose_frame_bytes(P0, P1);
  if (work_bytes < fixed + 2 * per)
    return set_error(ZR_EWORK, "zr_dose_filter: work buffer %zu < %zu", work_bytes, fixed + 2 * per);
  int chunk = (int)((work_bytes - fixed) / per);
  chunk &= ~1;
  if (chunk > N + (N & 1)) chunk = N + (N & 1);
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  const int K4 = zr_spectrum_pitch(P1);
  float2* ACC = (float2*)work;
  float2* T2 = ACC + (size_t)P0 * K4;
  float* FM = (float*)(T2 + (size_t)P0 * K4);
  float2* RW = (float2*)(FM + (size_t)P0 * K4);
  cudaStream_t st = (cudaStream_t)stream;
  for (int f0 = 0; f0 < N; f0 += chunk) {
    const int nfr = (N - f0) < chunk ? (N - f0) : chunk;
    const int npairs = (nfr + 1) / 2;
    ZR_DOSE_DISPATCH(P1, ZR_TRY((dose_rows<LL>(aligned, N, H, W, f0, npairs, K4, P0, RW, tw, st))));
    ZR_DOSE_DISPATCH(P0, ZR_TRY((dose_cols<LL>(RW, f0, nfr, K4, P1, *params, thres_q, dose_end, f0 == 0, ACC, FM,
                                                tw, st))));
  }
  ZR_DOSE_DISPATCH(P0, ZR_TRY((dose_icols<LL>(ACC, FM, params->normalize, K4, H, T2, tw, st))));
  // abs(IFFT2.execute(...)) at zorro.py:2484-2488: FFTW's inverse carries no 1/N
  const float scale = 1.0f;
  ZR_DOSE_DISPATCH(P1, ZR_TRY((dose_irows<LL>(T2, K4, H, W, scale, filt_sum, tw, st))));
  return ZR_OK;
}
