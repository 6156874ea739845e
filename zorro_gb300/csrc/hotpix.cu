// Gain correction and the outlier-pixel filter (hotpixFilter,
// zorro.py:2497-2672).  The host fits the normal CDF of the unaligned sum's
// histogram (zorro.py:2533-2592); the per-pixel parts run here and are folded
// into two maps so that every later kernel applies the filter while it reads
// a raw frame: corrected = hot_a * (gain * raw) + hot_b (zorro.py:2649).
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace zr {

// A running sum of floats as three floats hi + lo + lo2, by Knuth's two-sum
// (the exact error of an addition) on the sum and again on its errors, so that
// a thread's share of the float64 total needs no float64 operation per pixel:
// a converted addition a pixel kept the float64 pipe (2 lanes an SM) 79 % busy
// and bound the frame sum.  72 bits, so what is left is the rounding to float64
// at the end.  The terms are scaled by 2^-10 (exact) so that no sum of a few
// hundred of them overflows.
struct TripleSum {
  float hi = 0.0f, lo = 0.0f, lo2 = 0.0f;
  static __device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float t = __fadd_rn(a, b), d = __fsub_rn(t, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, d)), __fsub_rn(b, d));
    return t;
  }
  __device__ __forceinline__ void add(float v) {
    float e, e2;
    hi = two_sum(hi, v * 0.0009765625f, e);
    lo = two_sum(lo, e, e2);
    lo2 = __fadd_rn(lo2, e2);
  }
  // (an infinite or NaN sum has no error term)
  __device__ __forceinline__ double value() const {
    return 1024.0 * (fabsf(hi) < INFINITY ? (double)hi + ((double)lo + (double)lo2) : (double)hi);
  }
};

// Adds the CTA's share to the total.
__device__ __forceinline__ void add_total(double part, double* __restrict__ total) {
  for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x == 0 && total) {
    double v = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) v += red[i];
    atomicAdd(total, v);
  }
}

__global__ void k_gain_sum(FrameSrc f, float* __restrict__ sum, double* __restrict__ total) {
  const long long npix = (long long)f.H * f.W;
  double part = 0.0;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(p / f.W), x = (int)(p - (long long)y * f.W);
    float s = 0.0f;
    for (int n = 0; n < f.N; n++) s = __fadd_rn(s, load_corrected(f, n, y, x));
    sum[p] = s;
    part += (double)s;
  }
  add_total(part, total);
}

// Same sum, four pixels per thread (H*W % 4 == 0, aligned vector loads), the
// frames read GS_FRAMES at a time before any is added, so that each thread
// keeps that many loads in flight; the additions stay in frame order.
// Four CTAs an SM where a quad's eight loads fit 64 registers, three for
// float32: 40 K2 frames of uint16 228 us with three, 207 with four, 20 of
// float32 191 and 202.
constexpr int GS_FRAMES = 8;
__host__ __device__ constexpr int gs_ctas(int type) { return type == ZR_F32 ? 3 : 4; }

template <int TYPE>
__global__ void __launch_bounds__(256, gs_ctas(TYPE)) k_gain_sum_q(FrameSrc f, float* __restrict__ sum, double* __restrict__ total) {
  const long long n4 = (long long)f.H * f.W / 4;
  TripleSum part;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x) {
    const long long p = 4 * q;
    float4 g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (f.gain) g = __ldg(reinterpret_cast<const float4*>(f.gain + p));
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](const uint4& r) {
      float4 v = quad_value<TYPE>(r);
      if (f.gain) v = make_float4(__fmul_rn(g.x, v.x), __fmul_rn(g.y, v.y), __fmul_rn(g.z, v.z), __fmul_rn(g.w, v.w));
      if (f.gdiv != 0.0f)
        v = make_float4(__fdiv_rn(v.x, f.gdiv), __fdiv_rn(v.y, f.gdiv), __fdiv_rn(v.z, f.gdiv), __fdiv_rn(v.w, f.gdiv));
      s = make_float4(__fadd_rn(s.x, v.x), __fadd_rn(s.y, v.y), __fadd_rn(s.z, v.z), __fadd_rn(s.w, v.w));
    };
    uint4 r[GS_FRAMES];
    int n0 = 0;
    for (; n0 + GS_FRAMES <= f.N; n0 += GS_FRAMES) {
#pragma unroll
      for (int j = 0; j < GS_FRAMES; j++) r[j] = raw_quad<TYPE>(f.raw, (long long)(n0 + j) * f.fstride + p);
#pragma unroll
      for (int j = 0; j < GS_FRAMES; j++) add(r[j]);
    }
    if (n0 < f.N) {
#pragma unroll
      for (int j = 0; j < GS_FRAMES; j++)  // past the last frame: a repeated load, not added
        r[j] = raw_quad<TYPE>(f.raw, (long long)min(n0 + j, f.N - 1) * f.fstride + p);
#pragma unroll
      for (int j = 0; j < GS_FRAMES; j++)
        if (n0 + j < f.N) add(r[j]);
    }
    reinterpret_cast<float4*>(sum)[q] = s;
    part.add(s.x);
    part.add(s.y);
    part.add(s.z);
    part.add(s.w);
  }
  add_total(part.value(), total);
}

__global__ void k_histogram(const float* __restrict__ v, long long n, double e0, int nbins, unsigned int* __restrict__ counts) {
  extern __shared__ unsigned int hist[];
  for (int i = threadIdx.x; i < nbins; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    const double d = (double)v[p] - e0;
    if (d >= 0.0 && d <= (double)nbins) {
      int b = (int)floor(d);
      if (b == nbins) b = nbins - 1;  // the last bin is closed on the right
      atomicAdd(&hist[b], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nbins; i += blockDim.x)
    if (hist[i]) atomicAdd(counts + i, hist[i]);
}

// The same histogram when the first edge is k - 1/2 for an integer k (the
// hot-pixel bins, zorro.py:2530-2533), without float64: the bin of v is
// floor(v - k + 1/2) = floor(v) + [v - floor(v) >= 1/2] - k, exact in float32
// (v - floor(v) is exact for every float32 except just below zero, where the
// rounding cannot cross 1/2), and v equals the last edge exactly when that
// index is nbins and v - floor(v) is 1/2.
// Each warp counts in one of ``copies`` histograms in shared memory, which
// keeps the warps off each other's counters (a movie's sums fill a few tens
// of bins), and a thread reads 16 pixels before it counts any.
__global__ void __launch_bounds__(512) k_histogram_half(const float* __restrict__ v, long long n, int k, int nbins,
                                                        int copies, unsigned int* __restrict__ counts) {
  extern __shared__ unsigned int hist[];
  for (int i = threadIdx.x; i < nbins * copies; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  unsigned int* mine = hist + (threadIdx.x >> 5) % copies * nbins;
  auto count = [&](float x) {
    if (!(fabsf(x) < 1073741824.0f)) return;  // NaN, inf and values far outside every bin
    const float c = floorf(x);
    const float fr = x - c;
    int b = (int)c + (fr >= 0.5f ? 1 : 0) - k;
    if (b < 0 || b > nbins) return;
    if (b == nbins) {
      if (fr != 0.5f) return;
      b = nbins - 1;  // the last bin is closed on the right
    }
    atomicAdd(mine + b, 1u);
  };
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  if (((uintptr_t)v & 15) == 0) {
    const float4* q = reinterpret_cast<const float4*>(v);
    const long long n4 = n / 4;
    for (long long p = t; p < n4; p += 4 * step) {
      float4 x[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (p + i * step < n4) x[i] = __ldg(q + p + i * step);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (p + i * step < n4) {
          count(x[i].x);
          count(x[i].y);
          count(x[i].z);
          count(x[i].w);
        }
    }
    if (t < n - 4 * n4) count(__ldg(v + 4 * n4 + t));
  } else {
    for (long long p = t; p < n; p += step) count(__ldg(v + p));
  }
  __syncthreads();
  // many bins: several of a thread's loads in flight (200 x 180 sums in 20000
  // bins 11.2 us one by one, 7.1 so; 1024 x 1024 in 32000 50 and 20)
  if (copies == 1) {
#pragma unroll 8
    for (int i = threadIdx.x; i < nbins; i += 512)
      if (hist[i]) atomicAdd(counts + i, hist[i]);
    return;
  }
  for (int i = threadIdx.x; i < nbins; i += blockDim.x) {
    unsigned int c = 0;
    for (int j = 0; j < copies; j++) c += hist[j * nbins + i];
    if (c) atomicAdd(counts + i, c);
  }
}

__device__ __forceinline__ int rfl(int i, int n) { return i < 0 ? -i - 1 : (i >= n ? 2 * n - i - 1 : i); }

// The logistic exponents K (sigma - c relax), sigma = (s - mu) / sigma_fit, as
// A s + C with A = K / sigma_fit and C = -K c relax - A mu folded on the host
// in float64.  A pixel evaluates them with A and C split into float pairs, the
// product's and the sum's rounding errors kept: off by 2^-46 of the larger term
// at most, where a float64 multiply-add and its conversions kept the float64
// pipe 85 % busy.  The pairs serve while |C| < 2^17, where that is below 2^-29,
// out of sight of the exponentials' own roundings (40 K2 frames have a few tens;
// over 36 movies of 2 to 40 frames the maps' error against float64 is the same
// either way, 2.5e-8 to 2.8e-8 rms).  Beyond it, and for sums too large for the
// float products, float64, step by step when sigma_fit is 0.
struct HotConst {
  double rsig, A, C1, C2;
  float Ah, Al, C1h, C1l, C2h, C2l;
  float s_max;  // |s| below which the float pairs serve (0: none)
};

__device__ __forceinline__ float pair_fma(float Ah, float Al, float Ch, float Cl, float s) {
  const float p = __fmul_rn(Ah, s);
  const float e = __fmaf_rn(Al, s, __fmaf_rn(Ah, s, -p));
  const float t = __fadd_rn(p, Ch), b = __fsub_rn(t, p);
  const float r = __fadd_rn(__fsub_rn(p, __fsub_rn(t, b)), __fsub_rn(Ch, b));
  return __fadd_rn(t, __fadd_rn(r, __fadd_rn(e, Cl)));
}

// logisticMask and 1 - logisticMask of one pixel of the sum.
__device__ __forceinline__ void hot_mask(float s, const zr_hotpix_params_t& p, const HotConst& h, float& lm,
                                         float& conv) {
  float x1, x2;
  if (fabsf(s) < h.s_max) {
    x1 = pair_fma(h.Ah, h.Al, h.C1h, h.C1l, s);
    x2 = pair_fma(h.Ah, h.Al, h.C2h, h.C2l, s);
  } else if (h.rsig < INFINITY) {
    x1 = (float)fma(h.A, (double)s, h.C1);
    x2 = (float)fma(h.A, (double)s, h.C2);
  } else {
    const double sg = ((double)s - p.mu) * h.rsig, K = (double)p.logistic_k;
    x1 = (float)(K * (sg - (double)(p.cutoff_lower * p.relax)));
    x2 = (float)(K * (sg - (double)(p.cutoff_upper * p.relax)));
  }
  const float e1 = expf(x1);
  const float e2 = expf(x2);
  const float s1 = 1.0f / (1.0f + e1);
  lm = (1.0f - s1) / (1.0f + e2);
  if (lm < 0.5f || isinf(e2)) conv = 1.0f - lm;
  else conv = (e2 + s1) / (1.0f + e2);
}

// The maps for one tile of HF_TY x HF_TX pixels: a = logisticMask, and b, the
// PSF fill of singleton outliers plus neighbourFilt (zorro.py:2614-2649).
// Shared memory holds 1 - logisticMask on the tile and a two-pixel ring, the
// per-frame mean (sum / n_frames) and the neighbourly-outlier mask on a
// one-pixel ring; positions outside the image hold the values at the
// reflected positions, as scipy.ndimage.convolve(mode='reflect') reads them.
//   b = (1 - lm) * [nom <= thres] * psf(mean),  nom = (1 - lm) * psf(1 - lm),
// then for pixels with nom > thres the neighbour term is added: the mean of
// the per-frame means of the in-image 3 x 3 neighbours that are not in the
// mask (Python slicing: a window that starts at row or column -1 is empty),
// times 1 - lm, or bestMean when more than 66 % (or none but the pixel itself
// at 0.1 %) of the window is in the mask; float32 throughout, as np.mean of
// the float32 means and the float32 neighbourFilt array of the reference.
// The PSF sums keep the order of a per-pixel loop (taps row by row); a thread
// slides them down a strip of rows of one column.
// The dead and hot counts compare the float32 sum with s_dead / s_hot, the
// float32 values where the float64 quotient crosses the cut-offs (found on the
// host with the same float64 operations).
//
// Fused: the mask used to be a pass of its own (139 us for a K2 frame, bound
// by the float64 pipe) whose 1 - lm the fill read back per 32 x 32 tile (129
// us, 83 % of issue slots); together they take 160 us.
// Tiles of 8 rows where those of 32 leave SMs idle: what takes the time there is
// one tile's serial work (200 x 180: 13.2 us with 32 rows, 7.1 with 8; 512 x 512
// 13.2 and 10.8; at 1024 x 1024, 512 tiles of 32 rows, 18.6 with those).
constexpr int HF_SMS = 152;
constexpr int HF_TX = 64;
constexpr int HF_CW = HF_TX + 4;  // 1 - lm, two-pixel ring
constexpr int HF_MW = HF_TX + 2;  // mean and mask, one-pixel ring
constexpr int HF_T = 256;

// 3 x 3 sums down a column: ``psf_strip`` calls f(row, sum) for rows r0 .. r0 +
// n - 1, the sum of psf[3 a + b] src[row + 2 - a][col + 2 - b] in that order.
template <int PITCH, typename F>
__device__ __forceinline__ void psf_strip(const float* __restrict__ src, int r0, int n, const float (&k)[9], F f) {
  const float* q = src + r0 * PITCH;
  float t0 = q[2], t1 = q[1], t2 = q[0];                          // row r
  float m0 = q[PITCH + 2], m1 = q[PITCH + 1], m2 = q[PITCH];      // row r + 1
  for (int r = r0; r < r0 + n; r++) {
    q = src + (r + 2) * PITCH;
    const float u0 = q[2], u1 = q[1], u2 = q[0];
    float c = fmaf(k[0], u0, 0.0f);
    c = fmaf(k[1], u1, c);
    c = fmaf(k[2], u2, c);
    c = fmaf(k[3], m0, c);
    c = fmaf(k[4], m1, c);
    c = fmaf(k[5], m2, c);
    c = fmaf(k[6], t0, c);
    c = fmaf(k[7], t1, c);
    c = fmaf(k[8], t2, c);
    f(r, c);
    t0 = m0; t1 = m1; t2 = m2;
    m0 = u0; m1 = u1; m2 = u2;
  }
}

template <int HF_TY>
__global__ void __launch_bounds__(HF_T) k_hot_maps(const float* __restrict__ sum, int H, int W, int nfr,
                                                   zr_hotpix_params_t p, HotConst h, float s_dead, float s_hot,
                                                   float* __restrict__ LM, float* __restrict__ B,
                                                   unsigned int* __restrict__ counts) {
  constexpr int HF_CH = HF_TY + 4, HF_MH = HF_TY + 2;
  __shared__ float cv[HF_CH][HF_CW];
  __shared__ float mn[HF_MH][HF_MW];
  __shared__ uint8_t nm[HF_MH][HF_MW];
  const int ty0 = blockIdx.y * HF_TY, tx0 = blockIdx.x * HF_TX;
  const float fn = (float)nfr;
  const float bm = (float)p.best_mean;
  unsigned int dead = 0, hot = 0, nb = 0;
  float k[9];
#pragma unroll
  for (int i = 0; i < 9; i++) k[i] = p.psf[i];
  for (int e = threadIdx.x; e < HF_CH * HF_CW; e += HF_T) {
    const int ey = e / HF_CW, ex = e - (e / HF_CW) * HF_CW;
    const int y = ty0 + ey - 2, x = tx0 + ex - 2;
    const int gy = rfl(min(y, H + 1), H), gx = rfl(min(x, W + 1), W);
    const size_t g = (size_t)gy * W + gx;
    const float s = __ldg(sum + g);
    float lm, conv;
    hot_mask(s, p, h, lm, conv);
    cv[ey][ex] = conv;
    if (ey >= 1 && ey <= HF_MH && ex >= 1 && ex <= HF_MW) mn[ey - 1][ex - 1] = s / fn;
    if (ey >= 2 && ey < HF_TY + 2 && ex >= 2 && ex < HF_TX + 2 && y < H && x < W) {
      LM[g] = lm;
      dead += s < s_dead;
      hot += s >= s_hot;
    }
  }
  __syncthreads();
  // the mask on the tile and its ring (in-image positions only)
  constexpr int S1 = 3, N1 = (HF_MH + S1 - 1) / S1;  // strips of rows
  for (int e = threadIdx.x; e < HF_MW * S1; e += HF_T) {
    const int st = e / HF_MW, ex = e - st * HF_MW;
    const int gx = tx0 + ex - 1;
    psf_strip<HF_CW>(&cv[0][ex], st * N1, min(N1, HF_MH - st * N1), k, [&](int ey, float cc) {
      const int gy = ty0 + ey - 1;
      nm[ey][ex] = gy >= 0 && gy < H && gx >= 0 && gx < W && (cv[ey + 1][ex + 1] * cc) > p.neighbour_thres;
    });
  }
  __syncthreads();
  constexpr int N2 = HF_TY / (HF_T / HF_TX);  // rows a thread
  const int lx = threadIdx.x % HF_TX, x = tx0 + lx;
  if (x < W) {
    const int r0 = threadIdx.x / HF_TX * N2;
    psf_strip<HF_MW>(&mn[0][lx], r0, max(0, min(N2, H - ty0 - r0)), k, [&](int ly, float pm) {
      const int y = ty0 + ly;
      const float conv = cv[ly + 2][lx + 2];
      const bool neigh = nm[ly + 1][lx + 1] != 0;
      const float single = neigh ? 0.0f : conv;
      float bv = single * pm;
      if (neigh) {
        nb++;
        float nf;
        if (y == 0 || x == 0) {
          nf = bm;
        } else {
          const int y1 = min(y + 2, H), x1 = min(x + 2, W);
          int cnt = 0, size = 0, nk = 0;
          float sm = 0.0f;
          for (int yy = y - 1; yy < y1; yy++)
            for (int xx = x - 1; xx < x1; xx++) {
              size++;
              if (nm[yy - ty0 + 1][xx - tx0 + 1]) cnt++;
              else { sm += mn[yy - ty0 + 1][xx - tx0 + 1]; nk++; }
            }
          // cnt / size > 0.66 or <= 0.001 as integers: with size <= 9 no ratio
          // lies within 1/450 of 0.66, and cnt >= 1 (the pixel itself)
          if (50 * cnt > 33 * size || 1000 * cnt <= size) nf = bm;
          else nf = conv * (sm / (float)nk);
        }
        bv = bv + nf;
      }
      B[(size_t)y * W + x] = bv;
    });
  }
  for (int o = 16; o > 0; o >>= 1) {
    dead += __shfl_down_sync(0xffffffffu, dead, o);
    hot += __shfl_down_sync(0xffffffffu, hot, o);
    nb += __shfl_down_sync(0xffffffffu, nb, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (dead) atomicAdd(counts + 0, dead);
    if (hot) atomicAdd(counts + 1, hot);
    if (nb) atomicAdd(counts + 2, nb);
  }
}

// The float32 value t where the float64 test pred(s) = fn((double)s) changes
// from true (below t) to false: pred must be monotone over the float32
// values in their order (-inf ... -0, +0 ... +inf).  Returns the first value
// with pred false, +inf when pred holds up to +inf, NaN when it never holds
// and pred_never_true_means_nan.
static uint32_t order_key(float v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

static float key_value(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float v;
  memcpy(&v, &u, 4);
  return v;
}

template <class P>
static uint64_t first_false(P pred) {
  uint64_t a = order_key(-INFINITY), b = (uint64_t)order_key(INFINITY) + 1;
  while (a < b) {
    const uint64_t m = (a + b) / 2;
    if (pred(key_value((uint32_t)m))) a = m + 1;
    else b = m;
  }
  return a;
}

}  // namespace zr


using namespace zr;

extern "C" int zr_gain_sum(const zr_frames_t* frames, float* unaligned_sum, double* total, void* stream) {
  if (frames && frames->frame_movie)
    return set_error(ZR_EINVAL, "zr_gain_sum: one movie at a time (frame_movie must be NULL)");
  if (!frames || !frames->raw || !unaligned_sum) return set_error(ZR_EINVAL, "zr_gain_sum: null argument");
  FrameSrc f = make_src(frames);
  f.ha = nullptr;
  f.hb = nullptr;
  if (f.N <= 0 || f.H <= 0 || f.W <= 0) return set_error(ZR_EINVAL, "zr_gain_sum: empty movie");
  const long long npix = (long long)f.H * f.W;
  const int vec = f.type == ZR_U8 ? 4 : (f.type == ZR_F32 ? 16 : 8);  // bytes of one pixel quad
  if (npix % 4 == 0 && f.fstride % 4 == 0 && ((uintptr_t)unaligned_sum & 15) == 0 &&
      ((uintptr_t)f.raw % vec) == 0 && ((uintptr_t)f.gain & 15) == 0) {
    int blocks = (int)((npix / 4 + 255) / 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    cudaStream_t st = (cudaStream_t)stream;
    switch (f.type) {
      case ZR_U8: k_gain_sum_q<ZR_U8><<<blocks, 256, 0, st>>>(f, unaligned_sum, total); break;
      case ZR_U16: k_gain_sum_q<ZR_U16><<<blocks, 256, 0, st>>>(f, unaligned_sum, total); break;
      case ZR_F16: k_gain_sum_q<ZR_F16><<<blocks, 256, 0, st>>>(f, unaligned_sum, total); break;
      default: k_gain_sum_q<ZR_F32><<<blocks, 256, 0, st>>>(f, unaligned_sum, total);
    }
    return launched("k_gain_sum_q");
  }
  int blocks = (int)((npix + 255) / 256);
  if (blocks > 152 * 16) blocks = 152 * 16;
  k_gain_sum<<<blocks, 256, 0, (cudaStream_t)stream>>>(f, unaligned_sum, total);
  return launched("k_gain_sum");
}

extern "C" int zr_histogram(const float* values, long long n, double first_edge, int nbins, unsigned int* counts,
                            void* stream) {
  if (!values || !counts) return set_error(ZR_EINVAL, "zr_histogram: null argument");
  if (nbins <= 0 || nbins > 32768) return set_error(ZR_ESIZE, "zr_histogram: nbins %d outside [1, 32768]", nbins);
  int blocks = (int)((n + 1023) / 1024);
  if (blocks > 152 * 4) blocks = 152 * 4;
  if (blocks < 1) blocks = 1;
  const size_t smem = (size_t)nbins * sizeof(unsigned int);
  const double k = first_edge + 0.5;
  if (k == floor(k) && fabs(k) < 4194304.0) {
    // as many copies as 48 KB of shared memory holds, one a warp at most, and no
    // more counters than half a CTA's pixels, which have to be cleared and added
    // up: 1900 x 1900 sums of a mean of 20 in 3000 bins 8.3 us with one copy and
    // 10.3 with three, 200 x 180 in 1600 5.0 and 6.8 with seven; a K2 sum in
    // 46 takes 14.4 with sixteen
    const long long fit = 48 * 1024 / (long long)smem, worth = (n + blocks - 1) / blocks / nbins / 2;
    const int copies = (int)std::max(1LL, std::min({16LL, fit, worth}));
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k_histogram_half, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(smem * copies)), "hist attr"));
    k_histogram_half<<<blocks, 512, smem * copies, (cudaStream_t)stream>>>(values, n, (int)k, nbins, copies, counts);
    return launched("k_histogram_half");
  }
  ZR_TRY(cuda_check(cudaFuncSetAttribute(k_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "hist attr"));
  k_histogram<<<blocks, 512, smem, (cudaStream_t)stream>>>(values, n, first_edge, nbins, counts);
  return launched("k_histogram");
}

extern "C" int zr_hotpix_thresholds(double mu, double sigma, float cutoff_lower, float cutoff_upper, float* s_dead,
                                    float* s_hot) {
  if (!s_dead || !s_hot) return set_error(ZR_EINVAL, "zr_hotpix_thresholds: null argument");
  if (!(sigma >= 0.0)) return set_error(ZR_EINVAL, "zr_hotpix_thresholds: sigma %g is not >= 0", sigma);
  // sigma >= 0 makes (s - mu) / sigma monotone in s, so each cut-off test
  // changes its answer once along the float32 values
  const double cl = (double)cutoff_lower, cu = (double)cutoff_upper;
  const uint64_t end = (uint64_t)order_key(INFINITY) + 1;
  const uint64_t kd = first_false([&](float s) { return ((double)s - mu) / sigma < cl; });
  const uint64_t kh = first_false([&](float s) { return !(((double)s - mu) / sigma > cu); });
  *s_dead = kd >= end ? INFINITY : key_value((uint32_t)kd);  // +inf: only for an infinite cut-off
  *s_hot = kh >= end ? NAN : key_value((uint32_t)kh);         // NaN: no value is hot
  return ZR_OK;
}

extern "C" size_t zr_hotpix_work_bytes(int height, int width) {
  return (size_t)height * width * sizeof(float) + 256;
}

extern "C" int zr_hotpix_maps(const float* unaligned_sum, int height, int width, int n_frames,
                              const zr_hotpix_params_t* params, float* hot_a, float* hot_b, unsigned int* counts3,
                              void* work, size_t work_bytes, void* stream) {
  if (!unaligned_sum || !params || !hot_a || !hot_b || !counts3 || !work)
    return set_error(ZR_EINVAL, "zr_hotpix_maps: null argument");
  if (height < 4 || width < 4 || n_frames <= 0) return set_error(ZR_EINVAL, "zr_hotpix_maps: image too small");
  if (work_bytes < zr_hotpix_work_bytes(height, width))
    return set_error(ZR_EWORK, "zr_hotpix_maps: work buffer too small");
  const zr_hotpix_params_t p = *params;
  float s_dead = 0.0f, s_hot = 0.0f;
  ZR_TRY(zr_hotpix_thresholds(p.mu, p.sigma, p.cutoff_lower, p.cutoff_upper, &s_dead, &s_hot));
  HotConst h;
  const double Kd = (double)p.logistic_k;
  h.rsig = 1.0 / p.sigma;
  h.A = Kd * h.rsig;
  h.C1 = -(Kd * (double)(p.cutoff_lower * p.relax)) - h.A * p.mu;
  h.C2 = -(Kd * (double)(p.cutoff_upper * p.relax)) - h.A * p.mu;
  auto split = [](double v, float& hi, float& lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
  };
  split(h.A, h.Ah, h.Al);
  split(h.C1, h.C1h, h.C1l);
  split(h.C2, h.C2h, h.C2l);
  // (where |C| < 2^17 a larger |A s| only saturates; the products stay inside float's range)
  const double cmax = fmax(fabs(h.C1), fabs(h.C2));
  h.s_max = h.rsig < INFINITY && fabs(h.A) < 1e18 && cmax < 131072.0 ? 1e15f : 0.0f;
  const int nx = (width + HF_TX - 1) / HF_TX;
  auto run = [&](auto ty) {
    constexpr int TY = decltype(ty)::value;
    k_hot_maps<TY><<<dim3(nx, (height + TY - 1) / TY), HF_T, 0, (cudaStream_t)stream>>>(
        unaligned_sum, height, width, n_frames, p, h, s_dead, s_hot, hot_a, hot_b, counts3);
  };
  if ((long long)nx * ((height + 31) / 32) < HF_SMS) run(std::integral_constant<int, 8>());
  else run(std::integral_constant<int, 32>());
  return launched("k_hot_maps");
}
