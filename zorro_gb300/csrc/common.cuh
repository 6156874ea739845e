// Shared device-side helpers for the Zorro movie-registration kernels.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/zorro_gb300.h"
#include "fft_core.cuh"

namespace zr {

// One movie's frames as the kernels read them.  The corrected value of
// pixel (y, x) of frame n is
//     v = float32(gain[y,x] * raw[n,y,x])          (loadData, zorro.py:3466)
//     v = v / gdiv                                  (zorro.py:3477-3478, if gdiv != 0)
//     v = ha[y,x] * v + hb[y,x]                     (hotpixFilter, zorro.py:2649)
// with each step skipped when its pointer (or gdiv) is null/zero.
struct FrameSrc {
  const void* raw;
  int type;  // ZR_F32, ZR_U8, ZR_U16, ZR_F16
  const float* gain;
  const float* ha;
  const float* hb;
  float gdiv;
  int N, H, W;
  long long fstride;  // elements between consecutive frames
  const int* fmap;    // frame -> movie whose maps it reads (null: one map set)
  long long mstride;  // elements between the maps of consecutive movies
};

__host__ inline FrameSrc make_src(const zr_frames_t* f) {
  FrameSrc s;
  s.raw = f->raw;
  s.type = f->raw_type;
  s.gain = f->gain;
  s.ha = f->hot_a;
  s.hb = f->hot_b;
  s.gdiv = f->gain_divisor;
  s.N = f->n_frames;
  s.H = f->height;
  s.W = f->width;
  s.fstride = f->frame_stride ? f->frame_stride : (long long)f->height * f->width;
  s.fmap = f->frame_movie;
  s.mstride = f->frame_movie ? f->map_stride : 0;
  return s;
}

// Offset of frame n's gain and hot-pixel maps (the batched path's frames
// read the maps of their own movie).
__device__ __forceinline__ long long map_off(const FrameSrc& f, int n) {
  return f.fmap ? (long long)__ldg(f.fmap + n) * f.mstride : 0;
}

__device__ __forceinline__ float load_raw(const FrameSrc& f, long long idx) {
  switch (f.type) {
    case ZR_U8: return (float)__ldg((const uint8_t*)f.raw + idx);
    case ZR_U16: return (float)__ldg((const uint16_t*)f.raw + idx);
    case ZR_F16: return __half2float(__ldg((const __half*)f.raw + idx));
    default: return __ldg((const float*)f.raw + idx);
  }
}

__device__ __forceinline__ float load_corrected(const FrameSrc& f, int n, int y, int x) {
  const long long q = (long long)y * f.W + x;
  float v = load_raw(f, (long long)n * f.fstride + q);
  const long long p = q + map_off(f, n);
  if (f.gain) v = __fmul_rn(__ldg(f.gain + p), v);
  if (f.gdiv != 0.0f) v = __fdiv_rn(v, f.gdiv);
  if (f.ha) v = __fmaf_rn(__ldg(f.ha + p), v, __ldg(f.hb + p));
  return v;
}

// Raw bits of the four consecutive pixels at element i of the compile-time
// type TYPE (u8 in .x, u16/f16 in .x/.y, f32 in .x-.w; i a multiple of 4 and
// the array aligned for the vector load) and their values.
template <int TYPE>
__device__ __forceinline__ uint4 raw_quad(const void* raw, long long i) {
  uint4 r = make_uint4(0u, 0u, 0u, 0u);
  if (TYPE == ZR_U8) {
    r.x = __ldg(reinterpret_cast<const unsigned int*>((const uint8_t*)raw + i));
  } else if (TYPE == ZR_U16 || TYPE == ZR_F16) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>((const uint16_t*)raw + i));
    r.x = v.x;
    r.y = v.y;
  } else {
    r = __ldg(reinterpret_cast<const uint4*>((const float*)raw + i));
  }
  return r;
}

// Integers below 2^23 become floats by placing them in the mantissa of 2^23
// and subtracting it: exact, and on the FP32 pipe (conversions run at an
// eighth of its rate).
__device__ __forceinline__ float mantissa_value(unsigned int bits) { return __uint_as_float(bits) - 8388608.0f; }

template <int TYPE>
__device__ __forceinline__ float4 quad_value(const uint4 r) {
  constexpr unsigned int E = 0x4b000000u;  // 2^23
  if (TYPE == ZR_U8)
    return make_float4(mantissa_value(__byte_perm(r.x, E, 0x7440)), mantissa_value(__byte_perm(r.x, E, 0x7441)),
                       mantissa_value(__byte_perm(r.x, E, 0x7442)), mantissa_value(__byte_perm(r.x, E, 0x7443)));
  if (TYPE == ZR_U16)
    return make_float4(mantissa_value(__byte_perm(r.x, E, 0x7410)), mantissa_value(__byte_perm(r.x, E, 0x7432)),
                       mantissa_value(__byte_perm(r.y, E, 0x7410)), mantissa_value(__byte_perm(r.y, E, 0x7432)));
  if (TYPE == ZR_F16)
    return make_float4(__half2float(__ushort_as_half((unsigned short)(r.x & 0xffffu))),
                       __half2float(__ushort_as_half((unsigned short)(r.x >> 16))),
                       __half2float(__ushort_as_half((unsigned short)(r.y & 0xffffu))),
                       __half2float(__ushort_as_half((unsigned short)(r.y >> 16))));
  return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
}

// Corrected pixels (load_corrected) x = j + r STEP (r < 16) of row y of frame
// n: every load of the row's counts and maps is issued before any value is
// used.  The caller knows that the first FULL of them lie inside the row for
// every j; the others are loaded where x < cols and are 0 elsewhere.
template <int STEP, int FULL>
__device__ __forceinline__ void corrected16(const FrameSrc& f, int n, int y, int j, int cols, float* u) {
  const int lim = cols - j;
  const long long q = (long long)y * f.W + j;
  const long long p = q + map_off(f, n);
  const long long i = (long long)n * f.fstride + q;
  unsigned int bits[16];
  float g[16], a[16], b[16];
#define ZR_INSIDE(r) (r < FULL || r * STEP < lim)
  if (f.type == ZR_U8) {
#pragma unroll
    for (int r = 0; r < 16; r++) bits[r] = ZR_INSIDE(r) ? __ldg((const uint8_t*)f.raw + i + r * STEP) : 0u;
  } else if (f.type == ZR_F32) {
#pragma unroll
    for (int r = 0; r < 16; r++) bits[r] = ZR_INSIDE(r) ? __ldg((const unsigned int*)f.raw + i + r * STEP) : 0u;
  } else {
#pragma unroll
    for (int r = 0; r < 16; r++) bits[r] = ZR_INSIDE(r) ? __ldg((const uint16_t*)f.raw + i + r * STEP) : 0u;
  }
  if (f.gain) {
#pragma unroll
    for (int r = 0; r < 16; r++) g[r] = ZR_INSIDE(r) ? __ldg(f.gain + p + r * STEP) : 0.0f;
  }
  if (f.ha) {
#pragma unroll
    for (int r = 0; r < 16; r++) {
      a[r] = ZR_INSIDE(r) ? __ldg(f.ha + p + r * STEP) : 0.0f;
      b[r] = ZR_INSIDE(r) ? __ldg(f.hb + p + r * STEP) : 0.0f;
    }
  }
#undef ZR_INSIDE
  if (f.type == ZR_F32) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = __uint_as_float(bits[r]);
  } else if (f.type == ZR_F16) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = __half2float(__ushort_as_half((unsigned short)bits[r]));
  } else {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = (float)bits[r];
  }
  if (f.gain) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = __fmul_rn(g[r], u[r]);
  }
  if (f.gdiv != 0.0f) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = __fdiv_rn(u[r], f.gdiv);
  }
  if (f.ha) {
#pragma unroll
    for (int r = 0; r < 16; r++) u[r] = __fmaf_rn(a[r], u[r], b[r]);
  }
}

// Element i of the length-L complex sequence whose inverse FFT holds two real
// rows (row a in the real part, row b in the imaginary part), from the rows'
// half-plane spectra ``ra``/``rb`` (elements 0..L/2; null: a zero row):
// ga + i gb up to L/2, the Hermitian mirror conj(ga) + i conj(gb) above.
template <int L>
__device__ __forceinline__ float2 packed_rows(const float2* __restrict__ ra, const float2* __restrict__ rb, int i) {
  constexpr int half = L / 2;
  const int k = i <= half ? i : L - i;
  const float2 ga = ra ? __ldg(ra + k) : make_float2(0.0f, 0.0f);
  const float2 gb = rb ? __ldg(rb + k) : make_float2(0.0f, 0.0f);
  if (i == 0 || i == half) return make_float2(ga.x, gb.x);
  if (i < half) return make_float2(ga.x - gb.y, ga.y + gb.x);
  return make_float2(ga.x + gb.y, -ga.y + gb.x);
}

}  // namespace zr
