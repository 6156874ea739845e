// Tiled Fourier ring correlation (tiledFRC, zorro.py:2246-2310) and its
// rotational mean (rotmean, zorro_util.py:147-224).
//
// Each box x box tile of the even and odd sums is Hann-windowed; both real
// tiles go through one complex FFT per row (z = e + i o), the column pass
// transforms E and O and accumulates, per frequency and over all tiles, the
// normalised correlation real(E conj O) / sqrt(|O|^2 |E|^2) (float per tile
// and per group of FRC_TPG tiles, the groups summed in double).  The
// reference scales both spectra by 1/box^4 first; the ratio does not depend
// on that scale, so it is left out (it only risks float underflow).  Only
// kx in [0, box/2] is computed: the ratio at (-ky, -kx) equals the one at
// (ky, kx).
#include <math.h>

#include "common.cuh"
#include "internal.h"

namespace zr {

constexpr int FRC_NB = 4;
constexpr int FRC_TPG = 8;  // tiles accumulated per CTA of the column pass

// Hann window of apodization('hann', box): radius box/2, circular.  The
// squared radius is exact in float for power-of-two boxes.
__device__ __forceinline__ float hann_at(int y, int x, int B) {
  const float inv = 2.0f / (float)B;
  const float yy = (float)(y - B / 2) * inv, xx = (float)(x - B / 2) * inv;
  const float rr = xx * xx + yy * yy;
  return rr <= 1.0f ? 0.5f * (1.0f + cospif(sqrtf(rr))) : 0.0f;
}

// The window of one tile, computed once for all of them (a square root and a
// cosine a pixel; per tile they took most of the row pass's 372 us on a K2
// sum).
__global__ void k_frc_hann(int B, float* __restrict__ hann) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x < B) hann[y * B + x] = hann_at(y, x, B);
}

// Row pass: FRC_NB rows of one tile per CTA, bound by shared-memory bandwidth
// (73 %) and issue.  K2 sum, 144 tiles of 512 x 512: 372 -> 100 us with the
// window from k_frc_hann and no staging through shared memory on either side;
// the whole correlation 679 -> 290 us.  The first FFT pass reads the
// windowed pixels, the last one untangles E and O in registers.
template <int B>
__global__ void __launch_bounds__(fft_threads(B, FRC_NB), sm_minb(fft_threads(B, FRC_NB)))
    k_frc_rows(const float* __restrict__ even, const float* __restrict__ odd, const float* __restrict__ hann, int W,
               const int* __restrict__ offs, int K4, float2* __restrict__ RE, float2* __restrict__ RO,
               const float2* __restrict__ tw) {
  constexpr int T = fft_threads(B, FRC_NB);
  constexpr int RL = last_radix(B), NSL = B / RL;
  extern __shared__ float2 sm[];
  const int g = blockIdx.x, t = blockIdx.y;
  const int oy = offs[2 * t], ox = offs[2 * t + 1];
  block_fft_from<B, FRC_NB, T, -1, NSL>(sm, tw, [&](int r, int x) {
    const int y = g * FRC_NB + r;
    const size_t p = (size_t)(oy + y) * W + ox + x;
    const float h = __ldg(hann + y * B + x);
    return make_float2(__fmul_rn(h, __ldg(even + p)), __fmul_rn(h, __ldg(odd + p)));
  });
  const size_t base = ((size_t)t * (B / FRC_NB) + g) * K4 * FRC_NB;
  fft_last_paired<B, FRC_NB, T, -1>(sm, tw, [&](int r, int k0, const float2* x0, int k1, const float2* x1) {
    auto put = [&](int k, float2 zk, float2 zm) {
      const size_t o = base + k * FRC_NB + r;
      RE[o] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
      RO[o] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    };
#pragma unroll
    for (int q = 0; q < RL; q++) {
      const int m0 = k0 + q * NSL, m1 = k1 + q * NSL;
      if (m0 <= B / 2) put(m0, x0[q], k0 > 0 ? x1[RL - 1 - q] : x0[(RL - q) % RL]);
      if (m1 <= B / 2) put(m1, x1[q], k0 > 0 ? x0[RL - 1 - q] : x1[RL - 1 - q]);
    }
  });
  // the pitch's columns past B/2 are zero
  for (int e = (B / 2 + 1) * FRC_NB + threadIdx.x; e < K4 * FRC_NB; e += T)
    RE[base + e] = RO[base + e] = make_float2(0.0f, 0.0f);
}

// CTAs per SM that keep a T-thread CTA at <= 128 registers per thread
constexpr int frc_minblocks(int T) { return sm_minb(T); }

template <int B>
__global__ void __launch_bounds__(fft_threads(B, 2 * FRC_NB), frc_minblocks(fft_threads(B, 2 * FRC_NB)))
    k_frc_cols(const float2* __restrict__ RE, const float2* __restrict__ RO, int n_tiles, int K4,
               double* __restrict__ half, const float2* __restrict__ tw) {
  constexpr int T = fft_threads(B, 2 * FRC_NB);
  constexpr int LD = ld_of(B);
  constexpr int PER = (B * FRC_NB + T - 1) / T;
  extern __shared__ float2 sm[];
  const int k0 = blockIdx.x * FRC_NB;
  const int t0 = blockIdx.y * FRC_TPG;
  const int t1 = min(n_tiles, t0 + FRC_TPG);
  float acc[PER];  // at most FRC_TPG tiles per CTA; the groups are summed in double
#pragma unroll
  for (int i = 0; i < PER; i++) acc[i] = 0.0f;
  for (int t = t0; t < t1; t++) {
    const size_t tb = (size_t)t * (B / FRC_NB) * K4 * FRC_NB;
    // sequences 0 .. 3: columns k0 .. of E, 4 .. 7: of O
    block_fft_from<B, 2 * FRC_NB, T, -1>(sm, tw, [&](int b, int y) {
      const size_t i = tb + ((size_t)(y / FRC_NB) * K4 + k0 + b % FRC_NB) * FRC_NB + y % FRC_NB;
      return __ldg((b < FRC_NB ? RE : RO) + i);
    });
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int e = threadIdx.x + i * T;
      if (e < B * FRC_NB) {
        const int c = e / B, y = e - c * B;
        // the tile's correlation at this frequency in float (|r| <= 1, the
        // magnitudes taken separately so that their product cannot
        // overflow), the sum over tiles in double
        const float2 E = sm[c * LD + pidx(y)], O = sm[(FRC_NB + c) * LD + pidx(y)];
        const float num = fmaf(E.x, O.x, E.y * O.y);
        const float den = sqrtf(fmaf(O.x, O.x, O.y * O.y)) * sqrtf(fmaf(E.x, E.x, E.y * E.y));
        acc[i] += num / den;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const int e = threadIdx.x + i * T;
    if (e < B * FRC_NB) {
      const int c = e / B, y = e - c * B;
      half[((size_t)blockIdx.y * B + y) * K4 + k0 + c] = (double)acc[i];
    }
  }
}

// Sum over the tile groups and DC normalisation: the half plane V (double)
// and, fftshifted with its mirror, frc2d.
__global__ void k_frc_mean(const double* __restrict__ half, int ngroups, int B, int K4, double* __restrict__ V,
                           float* __restrict__ frc2d) {
  const int kx = blockIdx.x * blockDim.x + threadIdx.x, ky = blockIdx.y, hb = B / 2;
  if (kx > hb) return;
  const size_t plane = (size_t)B * K4, q = (size_t)ky * K4 + kx;
  double dc = 0.0, v = 0.0;
#pragma unroll 6
  for (int g = 0; g < ngroups; g++) {
    dc += half[g * plane];
    v += half[g * plane + q];
  }
  v = v / dc;
  V[q] = v;
  const int m = B - 1;
  frc2d[((ky + hb) & m) * B + ((kx + hb) & m)] = (float)v;
  if (kx > 0 && kx < hb) frc2d[((B - ky + hb) & m) * B + ((B - kx + hb) & m)] = (float)v;
}

// sqrt(n) - r (n < 2^20, |.| <= 1 within a ring), off by less than 2^-47: the float
// root h, the remainder e = n - h^2 (exact), x = sqrt(n) - h from 2 h x + x^2 = e as
// a float and what that leaves over, and Knuth's two-sum of h - r (exact) and x.
// A float64 square root is off by 2^-44 here.  One float64 addition, as with
// e / 2h alone, which is off by 2^-38; the square root itself took 7 us more for a
// K2 sum (a float64 operation keeps a warp's pipe 16 cycles).
__device__ __forceinline__ double root_minus(int n, int r) {
  if (n == 0) return -(double)r;
  const float h = sqrtf((float)n), g = 0.5f / h, e = fmaf(-h, h, (float)n);
  const float x = __fmul_rn(e, g), x2 = __fmul_rn(fmaf(-x, x, fmaf(-2.0f * h, x, e)), g);
  const float a = __fsub_rn(h, (float)r), t = __fadd_rn(a, x), b = __fsub_rn(t, a);
  const float err = __fadd_rn(__fsub_rn(a, __fsub_rn(t, b)), __fsub_rn(x, b));
  return (double)t + (double)__fadd_rn(err, x2);
}

// One ring r per CTA: pixels at radius rho in [r, r + 1) count with weight
// r + 1 - rho, those in [r - 1, r) with rho - r + 1 (the bilinear split of
// rotmean, gathered instead of scattered: no atomics), in float64.  A thread
// takes one line along the axis it crosses the ring by, where |that coordinate| is
// the larger one: four pixels a side at most
// (whole rows of a ring's top, of 60 pixels, kept their threads for 48 us; the
// scattered form with shared-memory atomics took 111 us).
constexpr int FRC_RT = 256;
__global__ void __launch_bounds__(FRC_RT) k_frc_rings(const double* __restrict__ V, int B, int K4,
                                                      double* __restrict__ frc) {
  __shared__ double red[2][FRC_RT / 32];
  const int r = blockIdx.x, hb = B / 2, m = B - 1;
  double s = 0.0, w = 0.0;
  for (int i = threadIdx.x; i < 2 * B; i += FRC_RT) {
    const bool swap = i >= B;  // lines of constant x, where |y| > |x|
    const int c = (swap ? i - B : i) - hb, c2 = c * c;
    const int hi2 = (r + 1) * (r + 1) - c2, lo2 = (r - 1) * (r - 1) - c2;
    int x0 = abs(c) + (swap ? 1 : 0);
    if (hi2 <= x0 * x0) continue;
    int x1 = (int)sqrtf((float)hi2) + 1;  // at least the last one inside, then exactly
    while (x1 * x1 >= hi2) x1--;
    if (r > 0 && lo2 > x0 * x0) {
      x0 = max(x0, (int)sqrtf((float)lo2) - 1);
      while (x0 * x0 < lo2) x0++;
    }
    for (int a = x0; a <= min(x1, hb); a++) {
      const int n = a * a + c2;
      const double d = root_minus(n, r);  // rho - r
      const double wt = n >= r * r ? 1.0 - d : 1.0 + d;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int x = q == 0 ? a : -a;
        if (x >= hb || (q == 1 && a == 0)) continue;
        const int ky = (swap ? x : c) & m, kx = (swap ? c : x) & m;
        const double v = kx <= hb ? V[(size_t)ky * K4 + kx] : V[(size_t)((B - ky) & m) * K4 + (B - kx)];
        s += v * wt;
        w += wt;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    w += __shfl_down_sync(0xffffffffu, w, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = s;
    red[1][threadIdx.x >> 5] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < FRC_RT / 32; i++) {
      s += red[0][i];
      w += red[1][i];
    }
    frc[r] = s / w;
  }
}

template <int B>
static int run_frc(const float* even, const float* odd, int W, const int* offs, int n_tiles, float* frc2d,
                   double* frc, int nout, void* work, cudaStream_t st) {
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  const int K4 = zr_spectrum_pitch(B);
  float2* RE = (float2*)work;
  float2* RO = RE + (size_t)n_tiles * B * K4;
  const int ngroups = (n_tiles + FRC_TPG - 1) / FRC_TPG;
  double* half = (double*)(RO + (size_t)n_tiles * B * K4);
  // the window waits in frc2d until the result replaces it
  k_frc_hann<<<dim3((B + 127) / 128, B), 128, 0, st>>>(B, frc2d);
  ZR_TRY(launched("k_frc_hann"));
  {
    constexpr int T = fft_threads(B, FRC_NB);
    const size_t smem = (size_t)FRC_NB * ld_of(B) * sizeof(float2);
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k_frc_rows<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "frc attr"));
    k_frc_rows<B><<<dim3(B / FRC_NB, n_tiles), T, smem, st>>>(even, odd, frc2d, W, offs, K4, RE, RO, tw);
    ZR_TRY(launched("k_frc_rows"));
  }
  {
    constexpr int T = fft_threads(B, 2 * FRC_NB);
    const size_t smem = (size_t)2 * FRC_NB * ld_of(B) * sizeof(float2);
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k_frc_cols<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "frc attr"));
    k_frc_cols<B><<<dim3(K4 / FRC_NB, ngroups), T, smem, st>>>(RE, RO, n_tiles, K4, half, tw);
    ZR_TRY(launched("k_frc_cols"));
  }
  double* V = (double*)RE;  // the row pass's output has been read
  k_frc_mean<<<dim3((B / 2 + 1 + 63) / 64, B), 64, 0, st>>>(half, ngroups, B, K4, V, frc2d);
  ZR_TRY(launched("k_frc_mean"));
  k_frc_rings<<<nout, FRC_RT, 0, st>>>(V, B, K4, frc);
  return launched("k_frc_rings");
}

}  // namespace zr

using namespace zr;

extern "C" size_t zr_frc_work_bytes(int n_tiles, int box) {
  const size_t K4 = zr_spectrum_pitch(box);
  const size_t ngroups = (n_tiles + FRC_TPG - 1) / FRC_TPG;
  return 2 * (size_t)n_tiles * box * K4 * sizeof(float2) + ngroups * box * K4 * sizeof(double);
}

extern "C" int zr_tiled_frc(const float* even, const float* odd, int height, int width, int box, const int* offsets,
                            int n_tiles, float* frc2d, double* frc, int nrings, void* work, size_t work_bytes,
                            void* stream) {
  if (!even || !odd || !offsets || !frc2d || !frc) return set_error(ZR_EINVAL, "zr_tiled_frc: null argument");
  if (n_tiles <= 0) return set_error(ZR_EINVAL, "zr_tiled_frc: no tiles (image smaller than the FRC box)");
  if (box != 128 && box != 256 && box != 512 && box != 1024)
    return set_error(ZR_ESIZE, "zr_tiled_frc: box %d not supported (128..1024, power of two)", box);
  const int nr_full = (int)ceil(sqrt((double)(box / 2) * (box / 2) * 2.0)) + 1;
  if (nrings <= 0 || nrings > nr_full) return set_error(ZR_EINVAL, "zr_tiled_frc: nrings must be in [1, %d]", nr_full);
  if (work_bytes < zr_frc_work_bytes(n_tiles, box))
    return set_error(ZR_EWORK, "zr_tiled_frc: work buffer %zu < %zu", work_bytes, zr_frc_work_bytes(n_tiles, box));
  (void)height;
  cudaStream_t st = (cudaStream_t)stream;
  switch (box) {
    case 128: return run_frc<128>(even, odd, width, offsets, n_tiles, frc2d, frc, nrings, work, st);
    case 256: return run_frc<256>(even, odd, width, offsets, n_tiles, frc2d, frc, nrings, work, st);
    case 512: return run_frc<512>(even, odd, width, offsets, n_tiles, frc2d, frc, nrings, work, st);
    default: return run_frc<1024>(even, odd, width, offsets, n_tiles, frc2d, frc, nrings, work, st);
  }
}
