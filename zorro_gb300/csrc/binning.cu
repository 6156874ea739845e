// Fourier binning: the sides' plans and the passes of every frame (binning.cuh).
#include <math.h>

#include "binning.cuh"

namespace zr {

static int bn_pow2_at_least(int v) {
  int m = 1;
  while (m < v) m <<= 1;
  return m;
}

// c_m = exp(i pi m^2 / n): m^2 is reduced mod 2n in integers, so the angle is
// exact before the (double) sincospi.
__device__ __forceinline__ float2 chirp(long long m, int n) {
  const long long q = (m * m) % (2LL * n);
  double s, c;
  sincospi((double)q / (double)n, &s, &c);
  return make_float2((float)c, (float)s);
}

// The chirp c[0 .. n) and the sequence that the outputs lo .. hi convolve
// with: c_m at m mod Q for lo - (n - 1) <= m <= hi, zero between.  (Over the
// whole GPU: one CTA's float64 pipe takes 250 us for 16384 of them.)
__global__ void k_bin_chirp(int n, int Q, int lo, int hi, float2* __restrict__ c, float2* __restrict__ seq) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) c[i] = chirp(i, n);
  if (i >= Q) return;
  float2 v = make_float2(0.0f, 0.0f);
  if (i <= hi) v = chirp(i, n);
  else if (i - Q >= lo - (n - 1)) v = chirp(Q - i, n);
  seq[i] = v;
}

// Its transform, in place.
template <int Q>
__global__ void __launch_bounds__(bn_threads(Q)) k_bin_plan(float2* __restrict__ seq, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  constexpr int T = bn_threads(Q);
  using P = Ip<Q>;
  ip_pass1<Q, 1, T, -1, false>(sm, [&](int, int j, float2* v) {
#pragma unroll
    for (int r = 0; r < 16; r++) v[r] = seq[j + r * P::A1];
  });
  __syncthreads();
  ip_pass2<Q, 1, T, -1, false>(sm, tw);
  ip_last<Q, 1, T, -1, false>(sm, tw, [&](int, int k, const float2* v) {
#pragma unroll
    for (int r = 0; r < P::RL; r++) seq[k + r * P::NS] = v[r];
  });
}

static int bn_plan(const BnSide& d, int lo, int hi, const float2* tw, cudaStream_t st) {
  if (d.n == d.Q) return ZR_OK;  // a direct transform: no chirp
  k_bin_chirp<<<(d.Q + 63) / 64, 64, 0, st>>>(d.n, d.Q, lo, hi, d.c, d.hat);
  ZR_TRY(launched("k_bin_chirp"));
  switch (d.Q) {
#define ZR_BN_PLAN(L)                                                                                        \
  case L:                                                                                                    \
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k_bin_plan<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                                           (int)bn_smem<L>()), "binning attr"));                             \
    k_bin_plan<L><<<1, bn_threads(L), bn_smem<L>(), st>>>(d.hat, tw);                                        \
    break;
    ZR_BN_PLAN(2048) ZR_BN_PLAN(4096) ZR_BN_PLAN(6144) ZR_BN_PLAN(8192) ZR_BN_PLAN(12288) ZR_BN_PLAN(16384)
#undef ZR_BN_PLAN
    default: return set_error(ZR_ESIZE, "binning convolution of %d points not supported", d.Q);
  }
  return launched("k_bin_plan");
}

// The sides that are taken: 513 .. 8192, or a longer one that a single CTA's
// shared memory holds directly.
static bool bn_long(int n) {
  return n == 9216 || n == 10240 || n == 11520 || n == 12288 || n == 15360 || n == 16384;
}
static bool bn_side_ok(int n) { return (n >= 2 && n <= 8192) || bn_long(n); }

// Scratch that a plan of side n is given.
static size_t bn_plan_elems(int n) { return (size_t)n + bn_pow2_at_least(2 * n - 1); }

}  // namespace zr

using namespace zr;

extern "C" size_t zr_bin_work_bytes(int H, int W, int Hb, int Wb) {
  const size_t Kb = (size_t)Wb / 2 + 1;
  const size_t plans = bn_plan_elems(W) + bn_plan_elems(H) + bn_plan_elems(Hb) + bn_plan_elems(Wb);
  return (plans + 2 * (size_t)H * Kb + 2 * (size_t)Hb * Kb) * sizeof(float2) + 256 * 8;
}

extern "C" int zr_bin_fourier(const zr_frames_t* frames, int Hb, int Wb, float* out, void* work, size_t work_bytes,
                              void* stream) {
  if (!frames || !frames->raw || !out || !work) return set_error(ZR_EINVAL, "zr_bin_fourier: null argument");
  FrameSrc f = make_src(frames);
  const int H = f.H, W = f.W;
  if (f.N <= 0 || H < 2 || W < 2) return set_error(ZR_EINVAL, "zr_bin_fourier: empty movie");
  if (Hb < 2 || Wb < 2 || (Hb & 1) || (Wb & 1) || Hb > H || Wb > W)
    return set_error(ZR_ESIZE, "zr_bin_fourier: binned shape %dx%d must be even and no larger than %dx%d", Hb, Wb,
                     H, W);
  if (!bn_side_ok(H) || !bn_side_ok(W) || !bn_side_ok(Hb) || !bn_side_ok(Wb) || Hb < 513 || Wb < 513)
    return set_error(ZR_ESIZE,
                     "zr_bin_fourier: frame %dx%d -> %dx%d: every side must be in 513..8192, or one of 9216, 10240, "
                     "11520, 12288, 15360, 16384 (binned sides at least 513)", H, W, Hb, Wb);
  // a long side's height is binned to no more than 8192 rows and (below 16384) no fewer than 2049
  if (bn_long(H) && ((H != 16384 && Hb <= 2048) || Hb > 8192))
    return set_error(ZR_ESIZE, "zr_bin_fourier: column lengths %d -> %d not supported", H, Hb);
  if (work_bytes < zr_bin_work_bytes(H, W, Hb, Wb))
    return set_error(ZR_EWORK, "zr_bin_fourier: work buffer %zu < %zu", work_bytes, zr_bin_work_bytes(H, W, Hb, Wb));
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  cudaStream_t st = (cudaStream_t)stream;
  const int Kb = Wb / 2 + 1, b0 = Hb / 2, b1 = Wb / 2;
  float2* w = (float2*)work;
  auto side = [&](int n, int K) {
    const BnSide d{n, bn_points(n, K), w, w + n};
    w += bn_plan_elems(n);
    return d;
  };
  const BnSide dw = side(W, 2 * b1 + 1), dh = side(H, 2 * b0 + 1), dhb = side(Hb, Hb), dwb = side(Wb, Wb);
  // 16-byte boundaries of the address space (``work`` itself is aligned to a
  // float2 only); zr_bin_work_bytes has the spare element of each
  auto even = [](float2* p) { return p + (((uintptr_t)p & 15) != 0); };
  float2* Ct = even(w);
  float2* Cc = Ct + (size_t)H * Kb;
  float2* Ci = even(Cc + (size_t)(Hb + 1) * Kb);
  ZR_TRY(bn_plan(dw, -b1, b1, tw, st));
  ZR_TRY(bn_plan(dh, -b0, b0, tw, st));
  ZR_TRY(bn_plan(dhb, 0, Hb - 1, tw, st));
  ZR_TRY(bn_plan(dwb, 0, Wb - 1, tw, st));
  const float scale = (float)(1.0 / ((double)Hb * Wb));  // normConst, zorro.py:1881
  for (int n = 0; n < f.N; n++) {
    ZR_TRY(bn_rows(f, n, dw, Wb, Ct, tw, st));
    ZR_TRY(bn_cols(Ct, dh, Hb, Kb, Cc, tw, st));
    ZR_TRY(bn_icols(Cc, dhb, Kb, Wb, scale, Ci, tw, st));
    ZR_TRY(bn_irows(Ci, dwb, Hb, out + (size_t)n * Hb * Wb, tw, st));
  }
  return ZR_OK;
}
