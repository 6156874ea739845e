// Shift every frame and sum (applyShifts, zorro.py:1734-1808, with
// lanczosIndexedShift, zorro_util.py:341-379), plus the even/odd half sums of
// lazyFouRingCorr (zorro.py:2237-2238), in one pass over the raw frames.
//
// Frame n is rolled by (roll_y, roll_x) (np.roll: out[i] = in[i - shift],
// circular; the offsets are given reduced to [0, H) and [0, W)), then convolved with the separable 3x3 kernel ky (x) kx
// (scipy.ndimage.convolve: out[i] = sum_k w[k] in[i - k + 1], 'reflect'
// borders of the rolled frame).  Sums run over frames in order in float32,
// as np.sum(images, axis=0) does for a float32 stack.
#include "common.cuh"
#include "internal.h"

namespace zr {

#ifndef ZR_SS_MINB
#define ZR_SS_MINB 6
#endif
#ifndef ZR_SS_R
#define ZR_SS_R 2
#endif
constexpr int SS_TX = 128, SS_THR = 256;  // tile columns (4 a lane), threads
constexpr int SS_NCH = (SS_TX + 2 + 3 + 3) / 4;  // 4-pixel chunks that cover a halo row at any alignment
constexpr int SS_TW = 4 * SS_NCH + 4;            // tile pitch: a guard column before the first chunk
// the corrections a frame's pixels take, resolved at compile time
enum { SS_NONE = 0, SS_HOT = 1, SS_GAIN_HOT = 2, SS_ANY = 3 };

__device__ __forceinline__ int refl1(int i, int n) { return i < 0 ? -i - 1 : (i >= n ? 2 * n - i - 1 : i); }

// One raw value of the compile-time type TYPE, as float.
template <int TYPE>
__device__ __forceinline__ float raw_at(const void* raw, long long idx) {
  if constexpr (TYPE == ZR_U8) return (float)__ldg((const uint8_t*)raw + idx);
  if constexpr (TYPE == ZR_U16) return (float)__ldg((const uint16_t*)raw + idx);
  if constexpr (TYPE == ZR_F16) return __half2float(__ldg((const __half*)raw + idx));
  return __ldg((const float*)raw + idx);
}

template <int TYPE>
__device__ __forceinline__ float corrected_at(const FrameSrc& f, long long fo, long long p) {
  float v = raw_at<TYPE>(f.raw, fo + p);
  if (f.gain) v = __fmul_rn(__ldg(f.gain + p), v);
  if (f.gdiv != 0.0f) v = __fdiv_rn(v, f.gdiv);
  if (f.ha) v = __fmaf_rn(__ldg(f.ha + p), v, __ldg(f.hb + p));
  return v;
}

// A CTA owns a 128 x 8R output tile and walks the frames in order.  For each
// frame the corrected values of the tile and its one-pixel halo (at the
// rolled source pixels) go to shared memory; a warp then filters R rows, a
// lane four consecutive columns of them.  Each column's R + 2 horizontal
// 3-tap results are computed once and slid down its rows for the vertical
// taps (the same products and sums as tap by tap).  The sum stays in
// registers, the even and odd sums (HALVES: the lazy FRC reads them) in
// shared memory.
//
// With VEC (arrays aligned for vector loads), the source columns of a tile
// that the roll does not wrap are one contiguous run a row: a warp reads it
// in aligned 4-pixel chunks of the raw frame and the maps, one a lane (the two
// chunks past the 32nd go to other warps), corrects them in registers and
// stores them as they are, 16 bytes a thread.  A row's misalignment (0..3
// pixels) is resolved where the row is read: two or three 16-byte loads and a
// choice, the same for a whole warp, of which six of their values the four
// columns take.  The chunks that hold the image's first and last column also
// store its reflection beside it.  Wrapped tiles are read pixel by pixel.
// Both paths apply the same operations to every pixel.
//
// What bounds it: issue slots.  The arithmetic is 6 operations a pixel, the
// addressing was ten times that: so the rows' sources and alignments are
// worked out once a frame by one thread a row (a table in shared memory, a
// frame ahead), and which corrections apply is a template argument.
// 40 K2 frames (3838 x 3710 uint8, gain and hot-pixel maps) with their aligned
// frames: 2135 us with 64 x 16 tiles whose chunks were stored and summed pixel
// by pixel, 1438 us now; the half sums of 20 such frames 1071 -> 740 us.  Two
// rows a thread (40 registers, six CTAs an SM) against four: 1438 and 1523 us.
template <int TYPE, bool VEC, int MAPS, bool HALVES, int R>
__global__ void __launch_bounds__(SS_THR, ZR_SS_MINB)
    k_shift_sum(FrameSrc f, const zr_shift_t* __restrict__ sh, float* __restrict__ sum,
                float* __restrict__ even, float* __restrict__ odd, float* __restrict__ aligned) {
  constexpr int TY = R * (SS_THR / 32), TH = TY + 2;
  __shared__ __align__(16) float tile[TH][SS_TW];
  __shared__ __align__(16) float half_acc[HALVES ? 2 : 1][HALVES ? TY : 1][HALVES ? SS_TX : 4];  // even, odd frames
  // per tile row and frame parity: first chunk of its run (-1: not needed),
  // tile index of column x0 - 1
  __shared__ int2 rowt[2][TH];
  const int x0 = blockIdx.x * SS_TX, y0 = blockIdx.y * TY;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, ly0 = wid * R;
  const int H = f.H, W = f.W;
  const long long HW = (long long)H * W;
  const int x = x0 + 4 * lane;  // this lane's first column
  float4 acc[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    acc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (HALVES) {
      *reinterpret_cast<float4*>(&half_acc[0][ly0 + i][4 * lane]) = acc[i];
      *reinterpret_cast<float4*>(&half_acc[1][ly0 + i][4 * lane]) = acc[i];
    }
  }
  // the tile holds the image columns xf .. xl; column xf sits at index 4 + s
  // of its row (s: the row's misalignment), column x0 - 1 at 4 + s - edge
  const int edge = x0 == 0;
  const int xf = x0 - 1 + edge, xl = min(x0 + SS_TX, W - 1);
  const int ncol = xl - xf + 1;
  const bool last = xl == W - 1, inner = !edge && !last;
  // source column of image column xf; roll offsets arrive reduced to [0, H) and [0, W)
  auto first_col = [&](int roll_x) {
    const int c0 = xf - roll_x;
    return c0 < 0 ? c0 + W : c0;
  };
  auto row_table = [&](int n) {
    const int i = threadIdx.x;
    if (i >= TH) return;
    const int gy = y0 - 1 + i, c0 = first_col(sh[n].roll_x);
    int2 r = make_int2(-1, 4 - edge);
    if (gy <= H) {
      int sy = refl1(gy, H) - sh[n].roll_y;
      if (sy < 0) sy += H;
      if (VEC && c0 + ncol <= W) {
        const int p0 = sy * W + c0;
        r.x = p0 & ~3;
        r.y += p0 & 3;
      } else {
        r.x = sy;
      }
    }
    rowt[n & 1][i] = r;
  };
  row_table(0);
  __syncthreads();
  const int nrow = min(R, H - (y0 + ly0));              // output rows of this warp inside the image
  const bool pairs = x + 4 <= W && (W & 1) == 0;        // rows start on 8 bytes
  for (int n = 0; n < f.N; n++) {
    const zr_shift_t t = sh[n];
    const long long fo = (long long)n * f.fstride;
    const int c0 = first_col(t.roll_x);
    const int par = n & 1;
    if (VEC && c0 + ncol <= W) {
      auto chunk = [&](int i, int k) {
        const int2 rt = rowt[par][i];
        const int run = rt.y - 4 + edge;  // misalignment s
        if (rt.x < 0 || 4 * k >= run + ncol) return;
        const int a = rt.x + 4 * k;
        float4 r;
        if (a + 4 <= HW) {
          r = quad_value<TYPE>(raw_quad<TYPE>(f.raw, fo + a));
          if (MAPS == SS_GAIN_HOT || (MAPS == SS_ANY && f.gain)) {
            const float4 g = __ldg(reinterpret_cast<const float4*>(f.gain + a));
            r = make_float4(__fmul_rn(g.x, r.x), __fmul_rn(g.y, r.y), __fmul_rn(g.z, r.z), __fmul_rn(g.w, r.w));
          }
          if (MAPS == SS_ANY && f.gdiv != 0.0f)
            r = make_float4(__fdiv_rn(r.x, f.gdiv), __fdiv_rn(r.y, f.gdiv), __fdiv_rn(r.z, f.gdiv),
                            __fdiv_rn(r.w, f.gdiv));
          if (MAPS == SS_GAIN_HOT || MAPS == SS_HOT || (MAPS == SS_ANY && f.ha)) {
            const float4 A = __ldg(reinterpret_cast<const float4*>(f.ha + a));
            const float4 B = __ldg(reinterpret_cast<const float4*>(f.hb + a));
            r = make_float4(__fmaf_rn(A.x, r.x, B.x), __fmaf_rn(A.y, r.y, B.y), __fmaf_rn(A.z, r.z, B.z),
                            __fmaf_rn(A.w, r.w, B.w));
          }
        } else {  // the chunk runs past the end of the frame: its pixels inside
          r.x = corrected_at<TYPE>(f, fo, a);
          r.y = a + 1 < HW ? corrected_at<TYPE>(f, fo, a + 1) : 0.0f;
          r.z = a + 2 < HW ? corrected_at<TYPE>(f, fo, a + 2) : 0.0f;
          r.w = 0.0f;
        }
        float* dst = &tile[i][4 + 4 * k];
        *reinterpret_cast<float4*>(dst) = r;
        if (inner) return;
        if (edge && k == 0)  // column -1 reads column 0
          dst[run - 1] = run == 0 ? r.x : (run == 1 ? r.y : (run == 2 ? r.z : r.w));
        const int e = run + ncol - 1 - 4 * k;  // column W - 1, when this chunk holds it
        if (last && e < 4) dst[e + 1] = e == 0 ? r.x : (e == 1 ? r.y : (e == 2 ? r.z : r.w));
      };
#pragma unroll
      for (int i = 0; i < (TH + 7) / 8; i++)
        if (wid + 8 * i < TH) chunk(wid + 8 * i, lane);
      // (from the last warp down: the first ones have the odd rows)
      const int e = SS_THR - 1 - threadIdx.x;
      if (e < 2 * TH) chunk(e >> 1, 32 + (e & 1));
    } else {
      for (int e = threadIdx.x; e < TH * (SS_TX + 2); e += SS_THR) {
        const int i = e / (SS_TX + 2), j = e - i * (SS_TX + 2);
        const int sy = rowt[par][i].x;
        if (sy < 0 || j >= ncol) continue;
        int sx = c0 + j;
        if (sx >= W) sx -= W;
        const float v = corrected_at<TYPE>(f, fo, (long long)sy * W + sx);
        tile[i][4 + j] = v;
        if (edge && j == 0) tile[i][3] = v;
        if (last && j == ncol - 1) tile[i][4 + j + 1] = v;
      }
    }
    __syncthreads();
    if (n + 1 < f.N) row_table(n + 1);
    // a function of columns x - 1 .. x + 4 of tile row ly0 + i
    auto six = [&](int i, auto g) {
      const int o = rowt[par][ly0 + i].y;
      const float4* q = reinterpret_cast<const float4*>(&tile[ly0 + i][4 * lane + (o & ~3)]);
      const float4 A = q[0], B = q[1];
      switch (o & 3) {
        case 0: return g(A.x, A.y, A.z, A.w, B.x, B.y);
        case 1: return g(A.y, A.z, A.w, B.x, B.y, B.z);
        case 2: return g(A.z, A.w, B.x, B.y, B.z, B.w);
        default: return g(A.w, B.x, B.y, B.z, B.w, reinterpret_cast<const float*>(q)[8]);
      }
    };
    float* out = aligned ? aligned + (size_t)n * HW + (size_t)(y0 + ly0) * W + x : nullptr;
    auto emit = [&](int i, float4 a) {
      acc[i] = make_float4(acc[i].x + a.x, acc[i].y + a.y, acc[i].z + a.z, acc[i].w + a.w);
      if (HALVES) {
        float4* h = reinterpret_cast<float4*>(&half_acc[par][ly0 + i][4 * lane]);
        const float4 v = *h;
        *h = make_float4(v.x + a.x, v.y + a.y, v.z + a.z, v.w + a.w);
      }
      if (out && i < nrow) {
        float* q = out + (size_t)i * W;
        if (pairs) {
          __stcs(reinterpret_cast<float2*>(q), make_float2(a.x, a.y));
          __stcs(reinterpret_cast<float2*>(q) + 1, make_float2(a.z, a.w));
        } else {
          if (x < W) __stcs(q, a.x);
          if (x + 1 < W) __stcs(q + 1, a.y);
          if (x + 2 < W) __stcs(q + 2, a.z);
          if (x + 3 < W) __stcs(q + 3, a.w);
        }
      }
    };
    if (t.apply) {
      auto hrow = [&](int i) {
        return six(i, [&](float a, float b, float c, float d, float e, float g) {
          return make_float4(fmaf(t.kx[0], c, fmaf(t.kx[1], b, t.kx[2] * a)),
                             fmaf(t.kx[0], d, fmaf(t.kx[1], c, t.kx[2] * b)),
                             fmaf(t.kx[0], e, fmaf(t.kx[1], d, t.kx[2] * c)),
                             fmaf(t.kx[0], g, fmaf(t.kx[1], e, t.kx[2] * d)));
        });
      };
      float4 h0 = hrow(0), h1 = hrow(1);
#pragma unroll
      for (int i = 0; i < R; i++) {
        const float4 h2 = hrow(i + 2);
        emit(i, make_float4(fmaf(t.ky[0], h2.x, fmaf(t.ky[1], h1.x, t.ky[2] * h0.x)),
                            fmaf(t.ky[0], h2.y, fmaf(t.ky[1], h1.y, t.ky[2] * h0.y)),
                            fmaf(t.ky[0], h2.z, fmaf(t.ky[1], h1.z, t.ky[2] * h0.z)),
                            fmaf(t.ky[0], h2.w, fmaf(t.ky[1], h1.w, t.ky[2] * h0.w))));
        h0 = h1;
        h1 = h2;
      }
    } else {
#pragma unroll
      for (int i = 0; i < R; i++)
        emit(i, six(i + 1, [](float, float b, float c, float d, float e, float) { return make_float4(b, c, d, e); }));
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < R; i++) {
    if (i >= nrow) continue;
    const size_t p = (size_t)(y0 + ly0 + i) * W + x;
    auto put = [&](float* dst, float4 a) {
      if (x < W) dst[p] = a.x;
      if (x + 1 < W) dst[p + 1] = a.y;
      if (x + 2 < W) dst[p + 2] = a.z;
      if (x + 3 < W) dst[p + 3] = a.w;
    };
    put(sum, acc[i]);
    if (HALVES) {
      if (even) put(even, *reinterpret_cast<const float4*>(&half_acc[0][ly0 + i][4 * lane]));
      if (odd) put(odd, *reinterpret_cast<const float4*>(&half_acc[1][ly0 + i][4 * lane]));
    }
  }
}

struct SsArgs {
  FrameSrc f;
  const zr_shift_t* shifts;
  float *sum, *even, *odd, *aligned;
  dim3 grid;
  cudaStream_t st;
};

template <int TYPE, bool VEC, int MAPS, int R>
static void launch_halves(const SsArgs& a, bool halves) {
  if (halves)
    k_shift_sum<TYPE, VEC, MAPS, true, (R > 2 ? 2 : R)><<<a.grid, SS_THR, 0, a.st>>>(a.f, a.shifts, a.sum, a.even, a.odd,
                                                                                  a.aligned);
  else
    k_shift_sum<TYPE, VEC, MAPS, false, R><<<a.grid, SS_THR, 0, a.st>>>(a.f, a.shifts, a.sum, a.even, a.odd, a.aligned);
}

template <int TYPE>
static void launch_shift(const SsArgs& a, bool vec, bool tall, bool halves, int maps) {
  constexpr int R = ZR_SS_R;
  if (!vec) {
    if (tall) launch_halves<TYPE, false, SS_ANY, R>(a, halves);
    else launch_halves<TYPE, false, SS_ANY, 1>(a, halves);
    return;
  }
  if (!tall) return launch_halves<TYPE, true, SS_ANY, 1>(a, halves);
  switch (maps) {
    case SS_NONE: return launch_halves<TYPE, true, SS_NONE, R>(a, halves);
    case SS_HOT: return launch_halves<TYPE, true, SS_HOT, R>(a, halves);
    case SS_GAIN_HOT: return launch_halves<TYPE, true, SS_GAIN_HOT, R>(a, halves);
    default: launch_halves<TYPE, true, SS_ANY, R>(a, halves);
  }
}

}  // namespace zr

using namespace zr;

extern "C" int zr_shift_sum(const zr_frames_t* frames, const zr_shift_t* shifts, float* image_sum, float* even_sum,
                            float* odd_sum, float* aligned, void* stream) {
  if (frames && frames->frame_movie)
    return set_error(ZR_EINVAL, "zr_shift_sum: one movie at a time (frame_movie must be NULL)");
  if (!frames || !frames->raw || !shifts || !image_sum) return set_error(ZR_EINVAL, "zr_shift_sum: null argument");
  FrameSrc f = make_src(frames);
  if (f.N <= 0 || f.H < 2 || f.W < 2) return set_error(ZR_EINVAL, "zr_shift_sum: empty movie");
  cudaStream_t st = (cudaStream_t)stream;
  // chunked reads: every array aligned for its 4-pixel vector load at any
  // pixel index that is a multiple of 4
  const int qbytes = f.type == ZR_U8 ? 4 : (f.type == ZR_F32 ? 16 : 8);
  // (and pixel indices that fit an int)
  const bool vec = (long long)f.H * f.W < (1LL << 31) - 1024 && f.fstride % 4 == 0 && ((uintptr_t)f.raw % qbytes) == 0 && ((uintptr_t)f.gain & 15) == 0 &&
                   ((uintptr_t)f.ha & 15) == 0 && ((uintptr_t)f.hb & 15) == 0;
  const bool halves = even_sum || odd_sum;
  // tiles of 32 rows (16 with the half sums, whose accumulators take shared
  // memory); of 8 rows where those would leave the SMs short of CTAs (each
  // CTA walks every frame, so a small image is bound by that walk)
  const int nx = (f.W + SS_TX - 1) / SS_TX;
  const int rows = halves ? 16 : 8 * ZR_SS_R;
  const bool tall = (long long)nx * ((f.H + rows - 1) / rows) >= 2 * 152;
  const dim3 grid(nx, tall ? (f.H + rows - 1) / rows : (f.H + 7) / 8);
  const int maps = f.gdiv != 0.0f ? SS_ANY
                   : f.gain       ? (f.ha ? SS_GAIN_HOT : SS_ANY)
                                  : (f.ha ? SS_HOT : SS_NONE);
  const SsArgs a{f, shifts, image_sum, even_sum, odd_sum, aligned, grid, st};
  switch (f.type) {
    case ZR_U8: launch_shift<ZR_U8>(a, vec, tall, halves, maps); break;
    case ZR_U16: launch_shift<ZR_U16>(a, vec, tall, halves, maps); break;
    case ZR_F16: launch_shift<ZR_F16>(a, vec, tall, halves, maps); break;
    case ZR_F32: launch_shift<ZR_F32>(a, vec, tall, halves, maps); break;
    default: return set_error(ZR_EINVAL, "zr_shift_sum: raw type %d", f.type);
  }
  return launched("k_shift_sum");
}
