// Fourier binning of a movie (binStack with binKernel='fourier',
// zorro.py:1826-1904): per frame, the H x W DFT, the corners kept to
// Hb x Wb (rows [0, Hb/2) and [H - Hb/2, H), columns likewise), times
// normConst = 1/(Hb Wb), the unscaled Hb x Wb inverse DFT, and its real part.
//
// Frame sizes are arbitrary (K2 super-resolution frames are 7676 x 7420).  A
// side whose length the in-place engine has (bn_direct: 2^a 3^b 5^c lengths
// that detectors and their binned frames use, 4096, 5760, 11520 ...) is
// transformed directly; any other length n is a chirp-z transform
// (Bluestein): with c_m = exp(i pi m^2/n),
//     X_k = conj(c_k) sum_j (x_j conj(c_j)) c_{k-j},
// a linear convolution done as a circular one of length M.  Only the K
// frequencies that the crop keeps are asked for, so M >= n + K - 1 is enough
// (12288 instead of 16384 points for the 8184-pixel side of a K3 frame binned
// to 4092).  An inverse DFT is the conjugate of the forward DFT of the
// conjugate.
//
// Passes (one frame at a time, scratch in ``work``), each one launch:
//   rows     two real rows per complex DFT of length W, split by Hermitian
//            symmetry, columns kx in [0, Wb/2] kept, written transposed
//                                                        -> Ct [Kb][H]
//   columns  DFT of length H, frequencies -Hb/2 .. Hb/2  -> Cc [Kb][Hb + 1]
//   columns  the real part that the reference's real() keeps made explicit
//            (the cropped spectrum's Nyquist row and column averaged with
//            their mirrors), inverse DFT of length Hb, times 1/(Hb Wb)
//                                                        -> Ci [Kb][Hb]
//   rows     two rows per complex inverse DFT of length Wb -> out [Hb][Wb]
//
// What bounds it: shared-memory bandwidth and issue slots at 16 warps an SM.
// Two K3 super-resolution frames (8184 x 11520 uint8 to 4092 x 5760): 5.81 ms
// with 16384-point convolutions for every side but the longest, products and
// transposes as passes of their own and the chirps made by one CTA; 1.85 ms
// now.
#pragma once
#include "common.cuh"
#include "fft_inplace.cuh"
#include "internal.h"

namespace zr {

// Threads: one 16-point butterfly of the first pass each, 512 at most.
__host__ __device__ constexpr int bn_threads(int L) { return L > 8192 ? 512 : (L / 16 + 31) / 32 * 32; }

// One side's transform: length n, run as Q points, directly (n == Q) or as a
// convolution with the chirp c and the transformed sequence hat.
struct BnSide {
  int n, Q;
  float2 *c, *hat;
};

inline bool bn_direct(int n) {
  for (int i = 0; i <= IP_LENGTHS; i++)
    if (ip_length(i) == n) return n >= 2048;
  return false;
}

// Points of the transform of an n-pixel side with K consecutive frequencies
// wanted.
inline int bn_points(int n, int K) {
  if (bn_direct(n)) return n;
  const int m[] = {2048, 4096, 6144, 8192, 12288, 16384};
  for (int v : m)
    if (v >= n + K - 1) return v;
  return 0;
}

// Forward DFT of length n: ``load(j, v)`` fills v[r] with the inputs i = j + r
// Q/16 (those with i >= n are not used), ``out(k, X_k)`` receives the
// frequencies lo <= k <= hi (lo <= 0).  ``out`` may write to ``s``.
template <int Q, bool CHIRP, bool ONE_BY_ONE = false, typename Load, typename Out>
__device__ __forceinline__ void bn_dft(float2* s, const BnSide& d, int lo, int hi, const float2* __restrict__ tw,
                                       Load load, Out out) {
  using P = Ip<Q>;
  constexpr int T = bn_threads(Q);
  if constexpr (CHIRP) {
    const float inv = 1.0f / (float)Q;
    auto put = [&](int k, float2 y) {
      const float2 v = cmulc(y, __ldg(d.c + (k < 0 ? -k : k)));
      out(k, make_float2(v.x * inv, v.y * inv));
    };
    ip_convolve<Q, T, ONE_BY_ONE>(
        s, tw, d.hat,
        [&](int j, float2* v) {
          load(j, v);
#pragma unroll
          for (int r = 0; r < 16; r++) {
            const int i = j + r * P::A1;
            v[r] = i < d.n ? cmulc(v[r], __ldg(d.c + i)) : make_float2(0.0f, 0.0f);
          }
        },
        [&](int j, const float2* v) {
#pragma unroll
          for (int r = 0; r < 16; r++) {
            const int i = j + r * P::A1;
            if (i <= hi) put(i, v[r]);
            else if (i - Q >= lo) put(i - Q, v[r]);
          }
        });
  } else {
    ip_pass1<Q, 1, T, -1, false, ONE_BY_ONE>(s, [&](int, int j, float2* v) { load(j, v); });
    __syncthreads();
    ip_pass2<Q, 1, T, -1, false>(s, tw);
    ip_last<Q, 1, T, -1, false, true>(s, tw, [&](int, int k, const float2* v) {
#pragma unroll
      for (int r = 0; r < P::RL; r++) {
        const int i = k + r * P::NS;
        if (i <= hi) out(i, v[r]);
        if (i - Q >= lo) out(i - Q, v[r]);  // (frequency n/2 is -n/2 too)
      }
    });
  }
}

// ``load`` of bn_dft from a function of the input's index.
template <int Q, typename F>
__device__ __forceinline__ auto bn_each(int n, F f) {
  return [=](int j, float2* v) {
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const int i = j + r * Ip<Q>::A1;
      v[r] = i < n ? f(i) : make_float2(0.0f, 0.0f);
    }
  };
}

// Runs the statements with the constants QQ (points) and CC (chirp-z or direct).
#define ZR_BN_CASE(L, ...) \
  case L: { constexpr int QQ = L; __VA_ARGS__; } break;
#define ZR_BN_DISPATCH(SIDE, ...)                                                                        \
  if ((SIDE).n == (SIDE).Q) {                                                                            \
    constexpr bool CC = false;                                                                           \
    switch ((SIDE).Q) {                                                                                  \
      ZR_BN_CASE(2048, __VA_ARGS__) ZR_BN_CASE(3072, __VA_ARGS__) ZR_BN_CASE(4096, __VA_ARGS__) ZR_BN_CASE(5120, __VA_ARGS__)        \
      ZR_BN_CASE(5760, __VA_ARGS__) ZR_BN_CASE(6144, __VA_ARGS__) ZR_BN_CASE(7680, __VA_ARGS__) ZR_BN_CASE(8192, __VA_ARGS__)        \
      ZR_BN_CASE(9216, __VA_ARGS__) ZR_BN_CASE(10240, __VA_ARGS__) ZR_BN_CASE(11520, __VA_ARGS__) ZR_BN_CASE(12288, __VA_ARGS__)     \
      ZR_BN_CASE(15360, __VA_ARGS__) ZR_BN_CASE(16384, __VA_ARGS__)                                                    \
      default: return set_error(ZR_ESIZE, "binning transform of %d points not supported", (SIDE).Q);     \
    }                                                                                                    \
  } else {                                                                                               \
    constexpr bool CC = true;                                                                            \
    switch ((SIDE).Q) {                                                                                  \
      ZR_BN_CASE(2048, __VA_ARGS__) ZR_BN_CASE(4096, __VA_ARGS__) ZR_BN_CASE(6144, __VA_ARGS__) ZR_BN_CASE(8192, __VA_ARGS__)        \
      ZR_BN_CASE(12288, __VA_ARGS__) ZR_BN_CASE(16384, __VA_ARGS__)                                                    \
      default: return set_error(ZR_ESIZE, "binning convolution of %d points not supported", (SIDE).Q);   \
    }                                                                                                    \
  }

template <int Q>
static size_t bn_smem() { return (size_t)ip_ld(Q, 1) * sizeof(float2); }

// The four passes (binning_rows.cu, binning_cols.cu, binning_icols.cu, binning_irows.cu)
int bn_rows(const FrameSrc& f, int n, const BnSide& d, int Wb, float2* Ct, const float2* tw, cudaStream_t st);
int bn_cols(const float2* Ct, const BnSide& d, int Hb, int Kb, float2* Cc, const float2* tw, cudaStream_t st);
int bn_icols(const float2* Cc, const BnSide& d, int Kb, int Wb, float scale, float2* Ci, const float2* tw,
             cudaStream_t st);
int bn_irows(const float2* Ci, const BnSide& d, int Hb, float* out, const float2* tw, cudaStream_t st);

}  // namespace zr
