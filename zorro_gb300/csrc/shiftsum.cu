// Shift every frame and sum (applyShifts, zorro.py:1734-1808, with
// lanczosIndexedShift, zorro_util.py:341-379), plus the even/odd half sums of
// lazyFouRingCorr (zorro.py:2237-2238), in one pass over the raw frames.
//
// Frame n is rolled by (roll_y, roll_x) (np.roll: out[i] = in[i - shift],
// circular; the offsets are given reduced to [0, H) and [0, W)), then convolved with the separable 3x3 kernel ky (x) kx
// (scipy.ndimage.convolve: out[i] = sum_k w[k] in[i - k + 1], 'reflect'
// borders of the rolled frame).  Sums run over frames in order in float32,
// as np.sum(images, axis=0) does for a float32 stack.
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace zr {

constexpr int SS_SMS = 152;
constexpr int SS_TX = 128, SS_THR = 256;  // tile columns (4 a lane), threads
constexpr int SS_NCH = (SS_TX + 2 + 3 + 3) / 4;  // 4-pixel chunks that cover a halo row at any alignment
constexpr int SS_TW = 4 * SS_NCH + 4;            // tile pitch: a guard column before the first chunk
constexpr int SS_NQ = (SS_TX + 2 + 31) / 32;     // columns a lane reads of a row pixel by pixel
// the corrections a frame's pixels take, resolved at compile time
// (SS_ANY: a gain divisor too; SS_BIG: any, and pixel offsets of more than 32 bits)
enum { SS_NONE = 0, SS_HOT = 1, SS_GAIN = 2, SS_GAIN_HOT = 3, SS_ANY = 4, SS_BIG = 5 };

__device__ __forceinline__ int refl1(int i, int n) { return i < 0 ? -i - 1 : (i >= n ? 2 * n - i - 1 : i); }

// Raw values of the compile-time type TYPE: their array, their bits, as float.
template <int TYPE>
__device__ __forceinline__ auto raw_ptr(const void* raw) {
  if constexpr (TYPE == ZR_U8) return (const uint8_t*)raw;
  else if constexpr (TYPE == ZR_F32) return (const unsigned int*)raw;
  else return (const unsigned short*)raw;
}
template <int TYPE, typename T>
__device__ __forceinline__ unsigned int raw_bits(const T* p) {
  return __ldg(p);
}
template <int TYPE>
__device__ __forceinline__ float bits_value(unsigned int b) {
  if constexpr (TYPE == ZR_F32) return __uint_as_float(b);
  else if constexpr (TYPE == ZR_F16) return __half2float(__ushort_as_half((unsigned short)b));
  else return (float)b;
}

template <int TYPE>
__device__ __forceinline__ float corrected_at(const FrameSrc& f, long long fo, long long p) {
  float v = bits_value<TYPE>(raw_bits<TYPE>(raw_ptr<TYPE>(f.raw) + fo + p));
  if (f.gain) v = __fmul_rn(__ldg(f.gain + p), v);
  if (f.gdiv != 0.0f) v = __fdiv_rn(v, f.gdiv);
  if (f.ha) v = __fmaf_rn(__ldg(f.ha + p), v, __ldg(f.hb + p));
  return v;
}

// A 4-pixel chunk's raw values and maps; a lane's columns of a row.
struct SsChunk {
  uint4 raw;
  float4 g, A, B;
};
template <int NQ>
struct SsRow {
  unsigned int v[NQ];
  float g[NQ], A[NQ], B[NQ];
};

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
// store its reflection beside it.  Wrapped tiles, and arrays not aligned so
// (frames of odd width), are read pixel by pixel, a row a warp with all of a
// lane's loads in flight: one at a time in a loop over the tile they took 654
// us instead of 423 for 23 float32 frames of 1709 x 2859 with hot-pixel maps.
// Their addresses are 32-bit byte offsets (64-bit ones were a quarter of the
// instructions; SS_BIG keeps them for frames of 2^30 pixels and more).
// Every path applies the same operations to every pixel.
//
// R = 1 serves images whose 8-row tiles all run at once.  The walk over the
// frames is what takes the time there, so the next frame's loads are in flight
// while this one is filtered (AHEAD, which also serves larger images that are
// read pixel by pixel: launch_shift): 40 frames of 512 x 512 with their aligned frames
// 83 us, 117 without; 27 of 302 x 114, 45 and 70.
//
// What bounds it: issue slots.  The arithmetic is 6 operations a pixel, the
// addressing was ten times that: so the rows' sources and alignments are
// worked out once a frame by one thread a row (a table in shared memory, a
// frame ahead), and which corrections apply is a template argument.
// 40 K2 frames (3838 x 3710 uint8, gain and hot-pixel maps) with their aligned
// frames: 2135 us with 64 x 16 tiles whose chunks were stored and summed pixel
// by pixel, 1360 us now; the half sums of 20 such frames 1071 -> 740 us.  Two
// rows a thread (40 registers, six CTAs an SM) against four: 1438 and 1523 us.
template <int TYPE, bool VEC, int MAPS, bool HALVES, int R, int CTAS, bool AHEAD>
__global__ void __launch_bounds__(SS_THR, CTAS)
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
  // where tile row i of a frame with shift t comes from: the row_table entry
  auto row_source = [&](int i, const zr_shift_t& t) {
    const int gy = y0 - 1 + i, c0 = first_col(t.roll_x);
    int2 r = make_int2(-1, 4 - edge);
    if (gy <= H) {
      int sy = refl1(gy, H) - t.roll_y;
      if (sy < 0) sy += H;
      if (VEC && c0 + ncol <= W) {
        const int p0 = sy * W + c0;
        r.x = p0 & ~3;
        r.y += p0 & 3;
      } else {
        r.x = sy;
      }
    }
    return r;
  };
  auto row_table = [&](int n) {
    const int i = threadIdx.x;
    if (i < TH) rowt[n & 1][i] = row_source(i, sh[n]);
  };
  row_table(0);
  __syncthreads();
  const int nrow = min(R, H - (y0 + ly0));              // output rows of this warp inside the image
  // rows of the aligned frames start on 8 bytes (any float-aligned buffer is taken)
  const bool pairs = x + 4 <= W && (W & 1) == 0 && (reinterpret_cast<uintptr_t>(aligned) & 7) == 0;
  constexpr int NR = (TH + 7) / 8;  // tile rows a warp reads
  static_assert(!(AHEAD && VEC), "pixel by pixel");
  const int extra = SS_THR - 1 - threadIdx.x;               // (from the last warp down: the first ones have the odd rows)
  const bool gain = MAPS == SS_GAIN || MAPS == SS_GAIN_HOT || (MAPS >= SS_ANY && f.gain);
  const bool hot = MAPS == SS_GAIN_HOT || MAPS == SS_HOT || (MAPS >= SS_ANY && f.ha);
  auto wraps = [&](const zr_shift_t& t) { return first_col(t.roll_x) + ncol > W; };
  // first pixel of chunk k of a row with source r, -1 where the row does not reach it
  auto first = [&](int2 r, int k) { return r.x < 0 || 4 * k >= r.y - 4 + edge + ncol ? -1 : r.x + 4 * k; };
  auto fetch = [&](long long fo, int a, SsChunk& q) {
    q.raw = raw_quad<TYPE>(f.raw, fo + a);
    if (gain) q.g = __ldg(reinterpret_cast<const float4*>(f.gain + a));
    if (hot) {
      q.A = __ldg(reinterpret_cast<const float4*>(f.ha + a));
      q.B = __ldg(reinterpret_cast<const float4*>(f.hb + a));
    }
  };
  auto value = [&](const SsChunk& q) {
    float4 r = quad_value<TYPE>(q.raw);
    if (gain) r = make_float4(__fmul_rn(q.g.x, r.x), __fmul_rn(q.g.y, r.y), __fmul_rn(q.g.z, r.z), __fmul_rn(q.g.w, r.w));
    if (MAPS >= SS_ANY && f.gdiv != 0.0f)
      r = make_float4(__fdiv_rn(r.x, f.gdiv), __fdiv_rn(r.y, f.gdiv), __fdiv_rn(r.z, f.gdiv), __fdiv_rn(r.w, f.gdiv));
    if (hot)
      r = make_float4(__fmaf_rn(q.A.x, r.x, q.B.x), __fmaf_rn(q.A.y, r.y, q.B.y), __fmaf_rn(q.A.z, r.z, q.B.z),
                      __fmaf_rn(q.A.w, r.w, q.B.w));
    return r;
  };
  auto tail = [&](long long fo, int a) {  // a chunk that runs past the end of the frame: its pixels inside
    return make_float4(corrected_at<TYPE>(f, fo, a), a + 1 < HW ? corrected_at<TYPE>(f, fo, a + 1) : 0.0f,
                       a + 2 < HW ? corrected_at<TYPE>(f, fo, a + 2) : 0.0f, 0.0f);
  };
  auto place = [&](int2 src, int i, int k, float4 r) {
    float* dst = &tile[i][4 + 4 * k];
    *reinterpret_cast<float4*>(dst) = r;
    if (inner) return;
    const int run = src.y - 4 + edge;  // misalignment s
    if (edge && k == 0)  // column -1 reads column 0
      dst[run - 1] = run == 0 ? r.x : (run == 1 ? r.y : (run == 2 ? r.z : r.w));
    const int e = run + ncol - 1 - 4 * k;  // column W - 1, when this chunk holds it
    if (last && e < 4) dst[e + 1] = e == 0 ? r.x : (e == 1 ? r.y : (e == 2 ? r.z : r.w));
  };
  // pixel (i, j) of the tile from its raw value and maps
  auto put = [&](int i, int j, float r, float g, float A, float B) {
    if (gain) r = __fmul_rn(g, r);
    if (MAPS >= SS_ANY && f.gdiv != 0.0f) r = __fdiv_rn(r, f.gdiv);
    if (hot) r = __fmaf_rn(A, r, B);
    tile[i][4 + j] = r;
    if (edge && j == 0) tile[i][3] = r;
    if (last && j == ncol - 1) tile[i][4 + j + 1] = r;
  };
  // A row pixel by pixel, wrapped or not: a lane takes every 32nd column (the
  // first lanes the last two), NQ of them from column 32 q0 on
  constexpr int NQ = VEC ? 2 : SS_NQ;  // (VEC: wrapped tiles are rare, registers are not)
  auto row_fetch = [&](auto wrap, long long fo, int c0, int sy, int q0, SsRow<NQ>& q) {
    using Off = std::conditional_t<MAPS == SS_BIG, unsigned long long, unsigned int>;  // bytes
    const int m = sy < 0 ? 0 : ncol - lane - 32 * q0;  // columns lane + 32 (q0 + i), 32 i < m
    const int c = c0 + lane + 32 * q0;
    const Off row = (Off)sy * W + c;
    const char* raw = reinterpret_cast<const char*>(raw_ptr<TYPE>(f.raw) + fo);
    auto map = [&](const float* p, Off o) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + o)); };
#pragma unroll
    for (int i = 0; i < NQ; i++) {
      const bool in = 32 * i < m;
      const Off e = row + 32 * i - (decltype(wrap)::value && c + 32 * i >= W ? W : 0), o = 4 * e;
      q.v[i] = in ? raw_bits<TYPE>(raw_ptr<TYPE>(raw + (Off)sizeof(*raw_ptr<TYPE>(nullptr)) * e)) : 0u;
      q.g[i] = in && gain ? map(f.gain, o) : 0.0f;
      q.A[i] = in && hot ? map(f.ha, o) : 0.0f;
      q.B[i] = in && hot ? map(f.hb, o) : 0.0f;
    }
  };
  auto row_place = [&](int sy, int i, int q0, const SsRow<NQ>& q) {
    const int m = sy < 0 ? 0 : ncol - lane - 32 * q0;
    if constexpr (VEC || AHEAD) {
#pragma unroll
      for (int j = 0; j < NQ; j++)
        if (32 * j < m) put(i, lane + 32 * (q0 + j), bits_value<TYPE>(q.v[j]), q.g[j], q.A[j], q.B[j]);
    } else {  // one branch a correction (503 us for ten frames of 3838 x 3711, pixel by pixel 639)
      float r[NQ];
#pragma unroll
      for (int j = 0; j < NQ; j++) r[j] = bits_value<TYPE>(q.v[j]);
      if (gain) {
#pragma unroll
        for (int j = 0; j < NQ; j++) r[j] = __fmul_rn(q.g[j], r[j]);
      }
      if (MAPS >= SS_ANY && f.gdiv != 0.0f) {
#pragma unroll
        for (int j = 0; j < NQ; j++) r[j] = __fdiv_rn(r[j], f.gdiv);
      }
      if (hot) {
#pragma unroll
        for (int j = 0; j < NQ; j++) r[j] = __fmaf_rn(q.A[j], r[j], q.B[j]);
      }
      float* dst = &tile[i][4 + lane + 32 * q0];
#pragma unroll
      for (int j = 0; j < NQ; j++)
        if (32 * j < m) dst[32 * j] = r[j];
      if (edge && lane == 0 && q0 == 0 && m > 0) dst[-1] = r[0];  // column -1 reads column 0
      if (last) {
#pragma unroll
        for (int j = 0; j < NQ; j++)
          if (32 * j + 1 == m) dst[32 * j + 1] = r[j];  // column W reads column W - 1
      }
    }
  };
  SsRow<NQ> rw[AHEAD ? NR : 1];
  auto load_ahead = [&](int n, const zr_shift_t& t) {
#pragma unroll
    for (int i = 0; i < NR; i++)
      row_fetch(std::true_type(), (long long)n * f.fstride, first_col(t.roll_x),
                wid + 8 * i < TH ? row_source(wid + 8 * i, t).x : -1, 0, rw[AHEAD ? i : 0]);
  };
  zr_shift_t t = sh[0], next = sh[min(1, f.N - 1)];
  if constexpr (AHEAD) load_ahead(0, t);
  for (int n = 0; n < f.N; n++) {
    if (!AHEAD) t = sh[n];
    const long long fo = (long long)n * f.fstride;
    const int c0 = first_col(t.roll_x);
    const int par = n & 1;
    if constexpr (AHEAD) {
#pragma unroll
      for (int i = 0; i < NR; i++) row_place(wid + 8 * i < TH ? rowt[par][wid + 8 * i].x : -1, wid + 8 * i, 0, rw[i]);
    } else if (!VEC || wraps(t)) {
      if (!VEC && wraps(t)) {
        for (int e = threadIdx.x; e < TH * (SS_TX + 2); e += SS_THR) {
          const int i = e / (SS_TX + 2), j = e - i * (SS_TX + 2);
          const int sy = rowt[par][i].x;
          if (sy < 0 || j >= ncol) continue;
          const long long p = (long long)sy * W + (c0 + j >= W ? c0 + j - W : c0 + j);
          put(i, j, bits_value<TYPE>(raw_bits<TYPE>(raw_ptr<TYPE>(f.raw) + fo + p)), gain ? __ldg(f.gain + p) : 0.0f,
              hot ? __ldg(f.ha + p) : 0.0f, hot ? __ldg(f.hb + p) : 0.0f);
        }
      } else {
#pragma unroll 1
        for (int i = wid; i < TH; i += SS_THR / 32) {
          const int sy = rowt[par][i].x;
#pragma unroll 1
          for (int q0 = 0; q0 < SS_NQ; q0 += NQ) {
            row_fetch(std::integral_constant<bool, VEC>(), fo, c0, sy, q0, rw[0]);
            row_place(sy, i, q0, rw[0]);
          }
        }
      }
    } else if constexpr (VEC) {
      auto one = [&](int i, int k) {
        const int2 src = rowt[par][i];
        const int a = first(src, k);
        if (a < 0) return;
        float4 r;
        if (a + 4 <= HW) {
          SsChunk q;
          fetch(fo, a, q);
          r = value(q);
        } else {
          r = tail(fo, a);
        }
        place(src, i, k, r);
      };
#pragma unroll
      for (int i = 0; i < NR; i++)
        if (wid + 8 * i < TH) one(wid + 8 * i, lane);
      if (extra < 2 * TH) one(extra >> 1, 32 + (extra & 1));
    }
    __syncthreads();
    if (n + 1 < f.N) {
      row_table(n + 1);
      if constexpr (AHEAD) load_ahead(n + 1, next);
    }
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
    if (AHEAD) {
      t = next;
      next = sh[min(n + 2, f.N - 1)];
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

template <int TYPE, bool VEC, int MAPS, int R, int CTAS, bool AHEAD = false>
static void launch_halves(const SsArgs& a, bool halves) {
  if (halves)
    k_shift_sum<TYPE, VEC, MAPS, true, R, CTAS, AHEAD><<<a.grid, SS_THR, 0, a.st>>>(a.f, a.shifts, a.sum, a.even,
                                                                                    a.odd, a.aligned);
  else
    k_shift_sum<TYPE, VEC, MAPS, false, R, CTAS, AHEAD><<<a.grid, SS_THR, 0, a.st>>>(a.f, a.shifts, a.sum, a.even,
                                                                                     a.odd, a.aligned);
}

// small: CTAs an SM of the kernel with tiles of 8 rows, 0 for those of 16.
//
// Frames read pixel by pixel: what a warp waits for are its loads, so it has the
// next frame's in flight while it filters (AHEAD), as far as the registers for
// them go: five columns of three rows, for the counts and for every map.  30
// frames of 1001 x 1003, microseconds: without maps 103 ahead (four CTAs an SM)
// and 164 not; of 901 x 903 with a gain 105 ahead (three) and 146 not, but just
// over one wave of those, 1001 x 1003, 158 and 148, until the fifth CTA an SM
// is full too: 1401 x 1403 252 and 282; with gain and hot-pixel maps (two) 97
// ahead at 701 x 703, where two are a wave, and 130 not, 184 and 169 at 1001 x
// 1003.
template <int TYPE>
static void launch_shift(const SsArgs& a, bool vec, int small, bool halves, int maps) {
  if (maps == SS_BIG) return launch_halves<TYPE, false, SS_BIG, 2, 5>(a, halves);
  if (small == 2) return launch_halves<TYPE, false, SS_ANY, 1, 2, true>(a, halves);
  if (small == 3) return launch_halves<TYPE, false, SS_ANY, 1, 3, true>(a, halves);
  if (vec) switch (maps) {
    case SS_NONE: return launch_halves<TYPE, true, SS_NONE, 2, 6>(a, halves);
    case SS_HOT: return launch_halves<TYPE, true, SS_HOT, 2, 6>(a, halves);
    case SS_GAIN: return launch_halves<TYPE, true, SS_GAIN, 2, 6>(a, halves);
    case SS_GAIN_HOT: return launch_halves<TYPE, true, SS_GAIN_HOT, 2, 6>(a, halves);
    default: return launch_halves<TYPE, true, SS_ANY, 2, 4>(a, halves);
  }
  const long long tiles = (long long)a.grid.x * a.grid.y;
  const bool two = tiles <= 2 * SS_SMS;
  switch (maps) {
    case SS_NONE: return launch_halves<TYPE, false, SS_NONE, 2, 4, true>(a, halves);
    case SS_GAIN:
      return tiles <= 3 * SS_SMS || tiles > 5 * SS_SMS ? launch_halves<TYPE, false, SS_GAIN, 2, 3, true>(a, halves)
                                                       : launch_halves<TYPE, false, SS_GAIN, 2, 5>(a, halves);
    case SS_HOT:
      return two ? launch_halves<TYPE, false, SS_HOT, 2, 2, true>(a, halves)
                 : launch_halves<TYPE, false, SS_HOT, 2, 5>(a, halves);
    case SS_GAIN_HOT:
      return two ? launch_halves<TYPE, false, SS_GAIN_HOT, 2, 2, true>(a, halves)
                 : launch_halves<TYPE, false, SS_GAIN_HOT, 2, 5>(a, halves);
    default: return launch_halves<TYPE, false, SS_ANY, 2, 5>(a, halves);
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
  const bool vec = f.fstride % 4 == 0 && ((uintptr_t)f.raw % qbytes) == 0 && ((uintptr_t)f.gain & 15) == 0 &&
                   ((uintptr_t)f.ha & 15) == 0 && ((uintptr_t)f.hb & 15) == 0;
  const bool halves = even_sum || odd_sum;
  // tiles of 16 rows; of 8, loading a frame ahead, where all of those run at
  // once, two an SM (registers for the loads) or else three: 20 frames of 75 x
  // 1031 34 us with two, 37 with three; 16 of 1665 x 167, 418 tiles, 43 us with
  // three, 53 with two, 59 as 16-row tiles; above one wave they lose (20 frames
  // of 1536 x 1536 266 us against 168)
  const int nx = (f.W + SS_TX - 1) / SS_TX;
  const bool big = (long long)f.H * f.W >= (1LL << 30);
  const long long tiles = (long long)nx * ((f.H + 7) / 8);
  const int small = big ? 0 : (tiles <= 2 * SS_SMS ? 2 : (vec && tiles <= 3 * SS_SMS ? 3 : 0));
  const dim3 grid(nx, small ? (f.H + 7) / 8 : (f.H + 15) / 16);
  // (byte offsets of pixels within 32 bits, for frames of less than 2^30)
  const int maps = big              ? SS_BIG
                   : f.gdiv != 0.0f ? SS_ANY
                   : f.gain         ? (f.ha ? SS_GAIN_HOT : SS_GAIN)
                                    : (f.ha ? SS_HOT : SS_NONE);
  const SsArgs a{f, shifts, image_sum, even_sum, odd_sum, aligned, grid, st};
  switch (f.type) {
    case ZR_U8: launch_shift<ZR_U8>(a, vec, small, halves, maps); break;
    case ZR_U16: launch_shift<ZR_U16>(a, vec, small, halves, maps); break;
    case ZR_F16: launch_shift<ZR_F16>(a, vec, small, halves, maps); break;
    case ZR_F32: launch_shift<ZR_F32>(a, vec, small, halves, maps); break;
    default: return set_error(ZR_EINVAL, "zr_shift_sum: raw type %d", f.type);
  }
  return launched("k_shift_sum");
}
