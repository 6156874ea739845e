// Peak search on the correlation windows (locatePeak, zorro.py:1099-1231).
//
// Each window is searched by one CTA, or by a cluster of them that share its rows
// out (k_peaks); a CTA keeps the w x w window in shared memory and runs, with all
// threads in lock step:
//   * suppressOrigin (zorro.py:1078-1083, literal stencil);
//   * Bmode 'opti': a bounded Brent minimisation over sigma in [0, 7] of
//     std(G_sigma*C) / (max - mean) (zorro.py:1108-1121).  The minimiser is
//     Brent's golden-section/parabolic method as published by Forsythe,
//     Malcolm and Moler (FMIN, 1977), the method behind scipy's
//     minimize_scalar(method='bounded'); each function value is a full
//     separable Gaussian filter of the window with 'reflect' borders and
//     radius int(4 sigma + 0.5), the filter scipy.ndimage.gaussian_filter
//     applies (axis 0, then axis 1);
//   * the maxShift circular mask, the argmax (first index on ties) and the
//     peak significance (zorro.py:1165-1168);
//   * the sub-pixel step: the 16 x 16 patch around the peak, its DFT,
//     zero-padded to 16*subPixReg and inverted, |.| and its argmax
//     (zorro.py:1180-1216), or the integer fallback at the window edge.
// Filtered values are recomputed on the fly in blocks of rows, so the CTA
// needs only the window and one row block of shared memory.
#include <cooperative_groups.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "fft_inplace.cuh"
#include "internal.h"

namespace zr {

namespace cg = cooperative_groups;

constexpr int PK_T = 1024;       // threads of a peak-search CTA
constexpr int PK_NW = PK_T / 32;  // warps
constexpr int PK_MAXR = 64;       // largest filter radius
constexpr int PK_SUBR = 8;        // +/- patch half-size (zorro.py:619)

// The bounded Brent search's state.  It lives in shared memory and only
// thread 0 touches it, so none of it stays in registers across the filter
// passes of the other threads.
struct BrentState {
  double a, b, fulc, nfc, xf, rat, e, x, fx, ffulc, fnfc, xm, tol1, tol2;
  int num;
};

struct PkShared {
  alignas(16) float wy[2 * PK_MAXR + 4];  // 16-byte aligned: read four taps at a time
  alignas(16) float wx[2 * PK_MAXR + 4];
  alignas(16) float ws[2 * PK_MAXR + 4];  // the search's weights, both axes
  float redf[PK_NW];
  int redi[PK_NW];
  float ws1[PK_NW], ws2[PK_NW], wmx[PK_NW];  // per-warp partials of the filter statistics
  int wcnt[PK_NW];
  double bc[4];
  int bi[2];
  double x;             // the Brent search's next abscissa
  int go;               // 1 while the search continues
  int r;                // filter radius of the current sigma
  int ry, rx;           // radii of the last filter
  BrentState bs;        // the search's state (thread 0 only)
};

__device__ __forceinline__ int reflect_idx(int i, int n) {
  while (i < 0 || i >= n) {
    if (i < 0) i = -i - 1;
    if (i >= n) i = 2 * n - i - 1;
  }
  return i;
}

// Gaussian weights exp(-0.5 k^2 / sigma^2), normalised (double, then float).
// One warp calls; returns the radius.  A dependent float64 operation takes 59
// cycles here, a division 570, a square root 590 and an exponential 1100, so
// what counts is the length of the chain: one exponential and one division
// for both taps +/- k, side by side on the lanes, and a shuffle tree for the
// sum (2 r + 1 additions in a row took up to 3400 cycles).
__device__ int gauss_weights(double sigma, float* w) {
  const int lane = threadIdx.x & 31;
  if (!(sigma > 1e-15)) {
    if (lane == 0) w[0] = 1.0f;
    return 0;
  }
  int r = (int)(4.0 * sigma + 0.5);
  if (r > PK_MAXR) r = PK_MAXR;
  const double c = -0.5 / (sigma * sigma);
  double e[(PK_MAXR + 32) / 32], s = 0.0;
#pragma unroll
  for (int i = 0; i < (PK_MAXR + 32) / 32; i++) {
    const int k = lane + 32 * i;
    e[i] = 0.0;
    if (32 * i <= r) {
      e[i] = k <= r ? exp(c * (double)k * (double)k) : 0.0;
      s += k == 0 ? e[i] : 2.0 * e[i];
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
  for (int i = 0; i < (PK_MAXR + 32) / 32; i++) {
    const int k = lane + 32 * i;
    if (k <= r) w[r - k] = w[r + k] = (float)(e[i] / s);
  }
  return r;
}

// Block reductions (all threads must call).

// max value with the smallest index among equal values; where no thread has
// one (all of them NaN), NaN and index 0, as np.argmax has it
__device__ void block_argmax(PkShared& sh, float& v, int& idx) {
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_down_sync(0xffffffffu, v, o);
    const int oi = __shfl_down_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sh.redf[wid] = v; sh.redi[wid] = idx; }
  __syncthreads();
  if (wid == 0) {
    v = lane < PK_NW ? sh.redf[lane] : -INFINITY;
    idx = lane < PK_NW ? sh.redi[lane] : 0x7fffffff;
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_down_sync(0xffffffffu, v, o);
      const int oi = __shfl_down_sync(0xffffffffu, idx, o);
      if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    if (lane == 0) {
      const bool none = idx == 0x7fffffff;
      sh.bc[3] = none ? nan("") : (double)v;
      sh.bi[0] = none ? 0 : idx;
    }
  }
  __syncthreads();
  v = (float)sh.bc[3];
  idx = sh.bi[0];
  __syncthreads();
}

// The reduction of every thread's v, on every thread.
template <typename Op>
__device__ float block_all(PkShared& sh, float v, Op op) {
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh.redf[threadIdx.x >> 5] = v;
  __syncthreads();
  v = sh.redf[threadIdx.x & 31];
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  return v;
}

struct FiltStats {
  double s1, s2;   // sum (f - c), sum (f - c)^2
  float mx;        // max f
  int n;
};

// Warp sums of the per-thread filter statistics (a shuffle tree in float),
// left in shared memory for stats_total.  All threads call.
__device__ __forceinline__ void stats_warps(PkShared& sh, float s1, float s2, int cnt, float mx) {
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sh.ws1[wid] = s1; sh.ws2[wid] = s2; sh.wcnt[wid] = cnt; sh.wmx[wid] = mx; }
}

// Their totals, the warps' partials summed in double in a fixed order (the
// float64 pipe only sees one warp's worth of additions).  Warp 0 calls, after
// a barrier; lane 0 holds the result.
__device__ __forceinline__ FiltStats stats_total(PkShared& sh) {
  const int lane = threadIdx.x & 31;
  FiltStats st;
  st.s1 = lane < PK_NW ? (double)sh.ws1[lane] : 0.0;
  st.s2 = lane < PK_NW ? (double)sh.ws2[lane] : 0.0;
  st.n = lane < PK_NW ? sh.wcnt[lane] : 0;
  st.mx = lane < PK_NW ? sh.wmx[lane] : -INFINITY;
  for (int o = 16; o > 0; o >>= 1) {
    st.s1 += __shfl_down_sync(0xffffffffu, st.s1, o);
    st.s2 += __shfl_down_sync(0xffffffffu, st.s2, o);
    st.n += __shfl_down_sync(0xffffffffu, st.n, o);
    st.mx = fmaxf(st.mx, __shfl_down_sync(0xffffffffu, st.mx, o));
  }
  return st;
}

// How the window's rows are laid out over the CTAs of a window's cluster and
// over their filter blocks, and which pixels each statistics thread sums.
//
// The statistics are float sums over the pixels of 1024 threads, in a fixed
// order that is part of the results (the Brent search takes its decisions on
// them): with w % 4 == 0 thread (ty, tx) = (t / (w/4), t % (w/4)) owns columns
// 4 tx .. 4 tx + 3 of the rows y with y mod (2 RB) = 2 ty, 2 ty + 1 (RB = 1024
// / (w/4)), otherwise thread (t / 64, t % 64) the columns tx + 64 i of the rows
// y mod 16 = ty; rows ascending, then columns.  A cluster of S CTAs gives
// each CTA a range of ty, hence runs of ``len`` rows from ``off`` in every
// ``period`` rows.  A single CTA takes blocks of consecutive rows.
struct PkRows {
  int w, period, off, len;  // row of run i, place j: i period + off + j
  int nruns, rpb;            // runs, runs per filter block
  int ty0, nty;              // ty range of this CTA
  int rb;                    // ty values (all CTAs)
  int cols;                  // tx values
  bool quad;                 // the w % 4 == 0 ownership
  bool direct;               // a block is one period of rows, a statistics thread's pixels are
                             // those of its horizontal unit and its neighbour's (w % 8 == 0)
  int pad, vp;               // reflected columns on each side of V, pitch of V
};

// V rows of a filter block: at most ``ROUNDS`` horizontal units (8 columns of
// a row) a thread, and what the shared memory beside the window holds.
__host__ __device__ inline int pk_vrows(int w, int vp, int rounds, int vfloats) {
  const int a = 2 * (rounds * PK_T / (2 * ((w + 7) / 8))), b = vfloats / vp;
  return a < b ? a : b;
}

__host__ __device__ inline bool pk_quad(int w) { return (w & 3) == 0 && w >= 16 && w <= 256; }
__host__ __device__ inline int pk_ty(int w) { return pk_quad(w) ? PK_T / (w / 4) : 16; }

template <int S>
__device__ __forceinline__ PkRows pk_rows(int w, int pad, int vfloats, int rank) {
  PkRows L;
  L.w = w;
  L.quad = pk_quad(w);
  L.rb = pk_ty(w);
  L.cols = L.quad ? w / 4 : 64;
  L.pad = pad;
  L.vp = ((w + 7) & ~7) + 2 * pad + 12;
  if (S == 1) {
    int nr = pk_vrows(w, L.vp, 1, vfloats);
    L.direct = L.quad && (w & 7) == 0 && nr >= min(2 * L.rb, w);
    if (L.direct) nr = 2 * L.rb;
    else if (nr > 8) nr &= ~7;
    if (nr > w) nr = w;
    L.period = L.len = nr;
    L.off = 0;
    L.nruns = (w + nr - 1) / nr;
    L.rpb = 1;
    L.ty0 = 0;
    L.nty = L.rb;
  } else {
    L.direct = false;
    const int m = L.quad ? 2 : 1;
    L.ty0 = rank * L.rb / S;
    L.nty = (rank + 1) * L.rb / S - L.ty0;
    L.period = m * L.rb;
    L.off = m * L.ty0;
    L.len = m * L.nty;
    L.nruns = (w + L.period - 1) / L.period;
    const int fit = pk_vrows(w, L.vp, 2, vfloats) / (m * ((L.rb + S - 1) / S));
    L.rpb = fit < L.nruns ? fit : L.nruns;
  }
  return L;
}

// R rows of one column through the vertical taps: acc[j] = sum_k wy[k]
// C[reflect(y + j + k - r)][x], k ascending.  The thread slides a window of R
// inputs: one 4-byte load (consecutive lanes, consecutive columns) and a
// broadcast weight (two in one load) feed R multiply-adds.
template <int R>
__device__ __forceinline__ void vcol(const float* __restrict__ C, int w, int x, int y, int r,
                                     const float* __restrict__ wy, float (&acc)[R]) {
  static_assert(R % 2 == 0, "weights are read in pairs");
  const int K = 2 * r + 1;
#pragma unroll
  for (int j = 0; j < R; j++) acc[j] = 0.0f;
  float d[R];
  auto taps = [&](auto in) {
#pragma unroll
    for (int j = 0; j < R - 1; j++) d[j] = in(j);
    auto tap = [&](int s, int k, float wk) {
      d[(s + R - 1) % R] = in(k + R - 1);
#pragma unroll
      for (int j = 0; j < R; j++) acc[j] = fmaf(wk, d[(s + j) % R], acc[j]);
    };
    int k = 0;
    for (; k + R <= K; k += R) {
#pragma unroll
      for (int s = 0; s < R; s += 2) {
        const float2 W = *reinterpret_cast<const float2*>(wy + k + s);
        tap(s, k + s, W.x);
        tap(s + 1, k + s + 1, W.y);
      }
    }
#pragma unroll
    for (int s = 0; s < R - 1; s++) {
      if (k + s >= K) break;
      tap(s, k + s, wy[k + s]);
    }
  };
  if (y >= r && y + R - 1 + r < w) {
    const float* p = C + (y - r) * w + x;
    taps([&](int i) { return p[i * w]; });
  } else if (r + R <= w) {  // one reflection at either edge
    taps([&](int i) {
      int q = y - r + i;
      q = q < 0 ? -1 - q : q;
      q = q < w ? q : 2 * w - 1 - q;
      return C[q * w + x];
    });
  } else {
    taps([&](int i) { return C[reflect_idx(y - r + i, w) * w + x]; });
  }
}

// 8 consecutive outputs of a filtered row: p + OFF is the input of tap 0 of
// output 0, p 16-byte aligned; taps in order.  A ring of 16 inputs in
// registers: one 16-byte load and four broadcast weights per 32
// multiply-adds.
template <int OFF>
__device__ __forceinline__ void hrow8(const float* __restrict__ p, const float* __restrict__ wx, int K, float (&f)[8]) {
  float v[16];
  auto load = [&](int at, const float* q) {
    const float4 t = *reinterpret_cast<const float4*>(q);
    v[at] = t.x;
    v[at + 1] = t.y;
    v[at + 2] = t.z;
    v[at + 3] = t.w;
  };
  load(0, p);
  load(4, p + 4);
  load(8, p + 8);
  auto taps = [&](int g, int q, float w) {  // tap 4 g + q of the ring's current turn
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = fmaf(w, v[(4 * g + OFF + q + j) % 16], f[j]);
  };
  int k = 0;
  for (; k + 16 <= K; k += 16) {
#pragma unroll
    for (int g = 0; g < 4; g++) {
      load((4 * g + 12) % 16, p + k + 4 * g + 12);
      const float4 W = *reinterpret_cast<const float4*>(wx + k + 4 * g);
      taps(g, 0, W.x);
      taps(g, 1, W.y);
      taps(g, 2, W.z);
      taps(g, 3, W.w);
    }
  }
#pragma unroll
  for (int g = 0; g < 4; g++) {
    if (k + 4 * g >= K) break;
    load((4 * g + 12) % 16, p + k + 4 * g + 12);
    const float4 W = *reinterpret_cast<const float4*>(wx + k + 4 * g);
    const int n = K - k - 4 * g;
    taps(g, 0, W.x);
    if (n > 1) taps(g, 1, W.y);
    if (n > 2) taps(g, 2, W.z);
    if (n > 3) taps(g, 3, W.w);
  }
}

// Vertical pass of a filter block (runs [r0, r0 + nr)) into V, with the
// columns that the horizontal taps reach beyond the edges written as their
// reflections.
template <int R>
__device__ __forceinline__ void vert_unit(const float* C, float* V, const PkRows& L, int r0, int run, int gg, int x,
                                          int ry, int rx, const float* wy) {
  const int w = L.w, y = (r0 + run) * L.period + L.off + gg * R;
  if (y >= w) return;
  float acc[R];
  vcol<R>(C, w, x, y, ry, wy, acc);
  float* out = V + (run * L.len + gg * R) * L.vp + L.pad + x;
  const int n = min(R, min(L.len - gg * R, w - y));
#pragma unroll
  for (int j = 0; j < R; j++)
    if (j < n) out[j * L.vp] = acc[j];
  auto mirror = [&](int q) {  // column q holds the same values
#pragma unroll
    for (int j = 0; j < R; j++)
      if (j < n) out[j * L.vp + q - x] = acc[j];
  };
  if (rx <= w) {
    if (x < rx) mirror(-1 - x);
    if (x >= w - rx) mirror(2 * w - 1 - x);
  } else {
    for (int m = -1 - rx / (2 * w); m <= 1 + rx / (2 * w); m++)
      for (int h = 0; h < 2; h++) {
        const int q = (h ? -1 - x : x) + 2 * w * m;  // reflect_idx(q) == x
        if (q != x && q >= -rx && q < w + rx) mirror(q);
      }
  }
}

template <int R>
__device__ __forceinline__ void vert_block(const float* C, float* V, const PkRows& L, int r0, int nr, int ry, int rx,
                                           const float* wy) {
  const int G = (L.len + R - 1) / R, units = L.w * G * nr;
  for (int u = threadIdx.x; u < units; u += PK_T) {
    const int g = u / L.w, x = u - g * L.w, run = g / G;
    vert_unit<R>(C, V, L, r0, run, g - run * G, x, ry, rx, wy);
  }
}

// Visit every filtered value of this CTA's rows.  MODE 0: statistics of all
// values.  MODE 1: masked statistics plus the argmax of (mask ? f : 0), first
// index on ties.  Each filter block of rows is filtered vertically into V,
// horizontally into registers, written over V as F and summed from there by
// the statistics threads in their own order.  Returns this statistics
// thread's sums.
struct PkSums {
  float s1, s2, mx, bv;
  int cnt, bi;
};

template <int MODE, int ROUNDS>
__device__ PkSums filter_rows(const float* C, float* V, const PkRows& L, int mS, int ry, int rx, const float* wy,
                              const float* wx, float c, bool use_mask) {
  const int w = L.w, U = (w + 7) / 8, K = 2 * rx + 1, OFF = (-rx) & 3;
  const int fp = 8 * U + 4;  // pitch of F
  PkSums a{0.0f, 0.0f, -INFINITY, -INFINITY, 0, 0x7fffffff};
  const int tl = threadIdx.x, tyl = tl / L.cols, tx = tl - tyl * L.cols, ty = L.ty0 + tyl;
  const bool owner = tyl < L.nty;
  // one pixel into the sums
  auto add = [&](int y, int x, float v) {
    bool in = true;
    if (MODE == 1) {
      const int dy = y - mS, dx = x - mS;
      in = !use_mask || (dy * dy + dx * dx < mS * mS);
      const float mv = in ? v : 0.0f;
      const int idx = y * w + x;
      if (mv > a.bv || (mv == a.bv && idx < a.bi)) { a.bv = mv; a.bi = idx; }
      a.cnt += in;
    }
    if (in) {
      const float d = v - c;
      a.s1 += d;
      a.s2 = fmaf(d, d, a.s2);
      a.mx = fmaxf(a.mx, v);
    }
  };
  if (MODE == 1 && ry == 0 && rx == 0) {  // no filter (the one weight is 1): the window's own values
    const int n = L.quad ? 2 : 1;
    for (int yb = n * ty; owner && yb < w; yb += n * L.rb)
      for (int y = yb; y < min(w, yb + n); y++) {
        const float* row = C + y * w;
        if (L.quad) {
          const float4 v = *reinterpret_cast<const float4*>(row + 4 * tx);
          add(y, 4 * tx, v.x);
          add(y, 4 * tx + 1, v.y);
          add(y, 4 * tx + 2, v.z);
          add(y, 4 * tx + 3, v.w);
        } else {
          for (int x = tx; x < w; x += 64) add(y, x, row[x]);
        }
      }
    return a;
  }
  auto horizontal = [&](int m, int x, float (&f)[8]) {
    const float* p = V + m * L.vp + L.pad + x - rx - OFF;
    switch (OFF) {
      case 0: hrow8<0>(p, wx, K, f); break;
      case 1: hrow8<1>(p, wx, K, f); break;
      case 2: hrow8<2>(p, wx, K, f); break;
      default: hrow8<3>(p, wx, K, f); break;
    }
  };
  if (ROUNDS == 1 && L.direct) {
    // thread t filters row 2 ty + (t & 1), columns 8 (tx / 2) .. + 7, and sums
    // rows 2 ty, 2 ty + 1, columns 4 tx .. + 3: half of what its lane
    // neighbour t ^ 1 holds, exchanged in registers
    const int G = (L.len + 7) / 8;
    const bool r8 = w * G <= PK_T;  // rows a thread filters vertically: 8, or 10 where that takes one round
    const int vg = threadIdx.x / w, vx = threadIdx.x - vg * w;
    const int m = 2 * ty + (tx & 1), x8 = 8 * (tx >> 1), odd = tx & 1;
    for (int r0 = 0; r0 < L.nruns; r0++) {
      if (r8) {
        if (vg < G) vert_unit<8>(C, V, L, r0, 0, vg, vx, ry, rx, wy);
      } else if (vg < (L.len + 9) / 10) {
        vert_unit<10>(C, V, L, r0, 0, vg, vx, ry, rx, wy);
      }
      __syncthreads();
      const int y0 = r0 * L.len;
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; j++) f[j] = 0.0f;
      if (owner && y0 + m < w) horizontal(m, x8, f);
      float fr[2][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? f[q] : f[4 + q], 1);
        fr[0][q] = odd ? got : f[q];
        fr[1][q] = odd ? f[4 + q] : got;
      }
      if (owner) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int y = y0 + 2 * ty + j;
          if (y >= w) break;
#pragma unroll
          for (int q = 0; q < 4; q++) add(y, 4 * tx + q, fr[j][q]);
        }
      }
      if (r0 + 1 < L.nruns) __syncthreads();  // V is read before it is written again
    }
    if (MODE == 0) a.cnt = threadIdx.x == 0 ? w * w : 0;
    return a;
  }
  for (int r0 = 0; r0 < L.nruns; r0 += L.rpb) {
    const int nr = min(L.rpb, L.nruns - r0);
    // rows a thread filters vertically: what splits the runs evenly
    const int e6 = (L.len + 5) / 6 * 6, e8 = (L.len + 7) / 8 * 8, e10 = (L.len + 9) / 10 * 10;
    if (ROUNDS == 1 || (e8 <= e6 && e8 <= e10)) vert_block<8>(C, V, L, r0, nr, ry, rx, wy);
    else if (e10 <= e6) vert_block<10>(C, V, L, r0, nr, ry, rx, wy);
    else vert_block<6>(C, V, L, r0, nr, ry, rx, wy);
    __syncthreads();
    // unit u: row 2 (u / 2U) + (u & 1), columns 8 ((u / 2) mod U) ...: neighbouring
    // lanes read rows whose pitch is 16 bytes mod 32, which spreads the
    // 32-byte column steps of the others over all banks
    const int rows = nr * L.len, units = ((rows + 1) & ~1) * U;
    float f[ROUNDS][8];
    auto unit = [&](int i, int& m, int& x) {
      const int u = threadIdx.x + i * PK_T, pr = (u >> 1) / U;
      m = 2 * pr + (u & 1);
      x = 8 * ((u >> 1) - pr * U);
      return u < units && m < rows;
    };
#pragma unroll
    for (int i = 0; i < ROUNDS; i++) {
      int m, x;
#pragma unroll
      for (int j = 0; j < 8; j++) f[i][j] = 0.0f;
      if (unit(i, m, x)) horizontal(m, x, f[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROUNDS; i++) {
      int m, x;
      if (unit(i, m, x)) {
        float4* F = reinterpret_cast<float4*>(V + m * fp + x);
        F[0] = make_float4(f[i][0], f[i][1], f[i][2], f[i][3]);
        F[1] = make_float4(f[i][4], f[i][5], f[i][6], f[i][7]);
      }
    }
    __syncthreads();
    auto sum_row = [&](int y, int m) {  // row y, at row m of F
      const float* F = V + m * fp;
      if (L.quad) {
        const float4 v = *reinterpret_cast<const float4*>(F + 4 * tx);
        add(y, 4 * tx, v.x);
        add(y, 4 * tx + 1, v.y);
        add(y, 4 * tx + 2, v.z);
        add(y, 4 * tx + 3, v.w);
      } else {
        for (int x = tx; x < w; x += 64) add(y, x, F[x]);
      }
    };
    if (owner) {
      const int per = L.quad ? 2 * L.rb : L.rb, n = L.quad ? 2 : 1;
      if (ROUNDS == 1) {  // rows y of [y0, y1) with y mod per in n ty .. n ty + n - 1
        const int y0 = r0 * L.len, y1 = min(w, y0 + L.len);
        for (int yb = y0 - y0 % per; yb < y1; yb += per)
          for (int j = 0; j < n; j++) {
            const int y = yb + n * ty + j;
            if (y >= y0 && y < y1) sum_row(y, y - y0);
          }
      } else {
        for (int i = 0; i < nr; i++)
          for (int j = 0; j < n; j++) {
            const int y = (r0 + i) * per + n * ty + j;
            if (y < w) sum_row(y, i * L.len + n * tyl + j);
          }
      }
    }
    if (r0 + L.rpb < L.nruns) __syncthreads();  // F is read before V is written again
  }
  if (MODE == 0) a.cnt = owner && tx == 0 && tyl == 0 && L.ty0 == 0 ? w * w : 0;
  return a;
}

// std(G_sigma * C) / (max - mean) from the statistics (zorro.py:1108-1121), in
// float64's own divisions and square root: the search branches on the value,
// and sums of squares beyond float32's range have to give infinity.  (Quotients
// and the root from reciprocal square roots and one remainder step, which are
// not always rounded so, took 149.0 us a lone window against 153.4, 643 against
// 648 for 190 K2 windows.)
__device__ __forceinline__ double objective(const FiltStats& st, float c, double n) {
  const double m1 = st.s1 / n;
  const double var = st.s2 / n - m1 * m1;
  const double mean = (double)c + m1;
  return sqrt(var > 0.0 ? var : 0.0) / ((double)st.mx - mean);
}

__device__ __forceinline__ double sgn1(double v) { return v > 0.0 ? 1.0 : (v < 0.0 ? -1.0 : 1.0); }

// Bounded Brent minimisation (FMM FMIN).  The search's state lives in shared
// memory and one thread steps it (brent_begin, brent_step): it leaves the next
// abscissa in sh.x with sh.go = 1, or the best one with sh.go = 0 and the
// number of function values in sh.bi[1].

// Thread 0: the next abscissa of the search (sh.x, sh.go = 1), or its end
// (sh.go = 0).
__device__ void brent_next(BrentState& S, PkShared& sh) {
  const double golden = 0.5 * (3.0 - sqrt(5.0));
  if (!(fabs(S.xf - S.xm) > (S.tol2 - 0.5 * (S.b - S.a)))) {
    sh.go = 0;
    return;
  }
  bool gstep = true;
  if (fabs(S.e) > S.tol1) {
    gstep = false;
    double r = (S.xf - S.nfc) * (S.fx - S.ffulc);
    double q = (S.xf - S.fulc) * (S.fx - S.fnfc);
    double p = (S.xf - S.fulc) * q - (S.xf - S.nfc) * r;
    q = 2.0 * (q - r);
    if (q > 0.0) p = -p;
    q = fabs(q);
    r = S.e;
    S.e = S.rat;
    if ((fabs(p) < fabs(0.5 * q * r)) && (p > q * (S.a - S.xf)) && (p < q * (S.b - S.xf))) {
      S.rat = (p + 0.0) / q;
      S.x = S.xf + S.rat;
      if (((S.x - S.a) < S.tol2) || ((S.b - S.x) < S.tol2)) S.rat = S.tol1 * sgn1(S.xm - S.xf);
    } else {
      gstep = true;
    }
  }
  if (gstep) {
    S.e = (S.xf >= S.xm) ? (S.a - S.xf) : (S.b - S.xf);
    S.rat = golden * S.e;
  }
  S.x = S.xf + sgn1(S.rat) * fmax(fabs(S.rat), S.tol1);
  sh.x = S.x;
  sh.go = 1;
}

__device__ double brent_first(double lo, double hi) { return lo + 0.5 * (3.0 - sqrt(5.0)) * (hi - lo); }

__device__ __forceinline__ void brent_tols(BrentState& S, double xatol3) {
  S.tol1 = sqrt(2.2e-16) * fabs(S.xf) + xatol3;
  S.tol2 = 2.0 * S.tol1;
}

__device__ void brent_begin(PkShared& sh, double lo, double hi, double xatol3, double x0, double f0) {
  BrentState S;
  S.a = lo;
  S.b = hi;
  S.fulc = S.nfc = S.xf = S.x = x0;
  S.rat = S.e = 0.0;
  S.fx = S.ffulc = S.fnfc = f0;
  S.num = 1;
  S.xm = 0.5 * (lo + hi);
  brent_tols(S, xatol3);
  brent_next(S, sh);
  if (!sh.go) {  // the search ended before its first step
    sh.x = S.xf;
    sh.bi[1] = S.num;
  }
  sh.bs = S;
}

__device__ void brent_step(PkShared& sh, double xatol3, int maxfun, double fu) {
  BrentState S = sh.bs;
  S.num += 1;
  if (fu <= S.fx) {
    if (S.x >= S.xf) S.a = S.xf; else S.b = S.xf;
    S.fulc = S.nfc; S.ffulc = S.fnfc;
    S.nfc = S.xf; S.fnfc = S.fx;
    S.xf = S.x; S.fx = fu;
  } else {
    if (S.x < S.xf) S.a = S.x; else S.b = S.x;
    if ((fu <= S.fnfc) || (S.nfc == S.xf)) {
      S.fulc = S.nfc; S.ffulc = S.fnfc;
      S.nfc = S.x; S.fnfc = fu;
    } else if ((fu <= S.ffulc) || (S.fulc == S.xf) || (S.fulc == S.nfc)) {
      S.fulc = S.x; S.ffulc = fu;
    }
  }
  S.xm = 0.5 * (S.a + S.b);
  brent_tols(S, xatol3);
  if (S.num >= maxfun) sh.go = 0;
  else brent_next(S, sh);
  if (!sh.go) {
    sh.x = S.xf;
    sh.bi[1] = S.num;
  }
  sh.bs = S;
}

// The sub-pixel step on a 16 x 16 filtered patch (zorro.py:1180-1216): its
// forward DFT (rows, then columns), the inverse DFT upsampled to an L x L
// grid (L = 16*sp, frequencies -8..7, unscaled like the reference's
// subIFFT2.execute()), |.| and its argmax (first index on ties).  ``scratch``
// holds 17*L float2 of shared memory.  All threads call.
//
// The L^2 values are sums of 16 terms each (L = 256: 1 M complex multiply-adds,
// 130 000 cycles, a third of a lone window's time).  They are computed by
// 16-point transforms instead, an eighth of the operations, which find every
// grid point that can hold the maximum; those few (one to four of a peak) are
// then summed term by term, and the argmax is taken among these values.  A
// value's error, of either way, is below 64 roundings of S = sum |F| (18 terms
// deep twice, or 2 x 4 butterfly stages and a twiddle), so the maximum's point
// lies within 4 x 64 of them of the largest value.  A lone
// window takes 146 us so instead of 211, 190 K2 windows 656 instead of 771.
constexpr float SUBPIX_MARGIN = 256.0f / 16777216.0f;

// cmul with its roundings spelled out: the same bits wherever it is inlined.
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ void subpix_search(const float* patch, int sp, const float2* __restrict__ tw, float2* scratch,
                              float2* patchF, PkShared& sh, float& bv, int& bi) {
  __shared__ float2 rowF[16 * 16];
  for (int e = threadIdx.x; e < 256; e += PK_T) {
    const int i = e >> 4, v = e & 15;
    float2 acc = make_float2(0.0f, 0.0f);
    for (int j = 0; j < 16; j++) {
      const float2 t = __ldg(tw + ((v * j) & 15) * (TWN / 16));
      acc.x = fmaf(patch[i * 16 + j], t.x, acc.x);
      acc.y = fmaf(patch[i * 16 + j], t.y, acc.y);
    }
    rowF[e] = acc;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 256; e += PK_T) {
    const int u = e >> 4, v = e & 15;
    float2 acc = make_float2(0.0f, 0.0f);
    for (int i = 0; i < 16; i++) acc = cadd(acc, cmul(rowF[i * 16 + v], __ldg(tw + ((u * i) & 15) * (TWN / 16))));
    patchF[e] = acc;
  }
  __syncthreads();
  // exp(+2 pi i m / L) for m in [0, L), after the L x 16 intermediate
  const int L = 16 * sp;
  const int tws = TWN / L;
  float2* Tx = scratch;
  float2* Wl = Tx + 16 * L;
  for (int m = threadIdx.x; m < L; m += PK_T) {
    float2 t = __ldg(tw + m * tws);
    t.y = -t.y;
    Wl[m] = t;
  }
  float fs = 0.0f;  // sum |F|, or more
  if (threadIdx.x < 256) fs = fabsf(patchF[threadIdx.x].x) + fabsf(patchF[threadIdx.x].y);
  const float S = block_all(sh, fs, [](float a, float b) { return a + b; });
  // Values near the maximum: outputs n = sp b + a of a transform of 16
  // frequencies f zero-padded to L are, for every a, a 16-point transform over
  // b of the inputs times exp(2 pi i f a / L).
  auto sixteenth = [&](const float2* in, int step, int a, float2 (&v)[16]) {
    const int up = a > 0 ? L : 0;  // a < sp: |f a| < L
#pragma unroll
    for (int f = 0; f < 16; f++) v[f] = cmul(in[f * step], Wl[f < 8 ? f * a : (f - 16) * a + up]);
    ip_dft<16, 1>(v);
  };
  if (threadIdx.x < 16 * sp) {
    const int a = threadIdx.x % sp, fy = threadIdx.x / sp;
    float2 v[16];
    sixteenth(patchF + 16 * fy, 1, a, v);
#pragma unroll
    for (int b = 0; b < 16; b++) Tx[fy * L + sp * b + a] = v[b];
  }
  __syncthreads();
  float most = 0.0f;  // largest |value|^2 of this thread's columns
  for (int e = threadIdx.x; e < L * sp; e += PK_T) {
    float2 v[16];
    sixteenth(Tx + e % L, L, e / L, v);
#pragma unroll
    for (int b = 0; b < 16; b++) most = fmaxf(most, fmaf(v[b].x, v[b].x, v[b].y * v[b].y));
  }
  const float M2 = block_all(sh, most, [](float a, float b) { return fmaxf(a, b); });
  bv = -INFINITY;
  bi = 0x7fffffff;
  int* list = reinterpret_cast<int*>(rowF);
  constexpr int CAP = sizeof(rowF) / sizeof(int);
  int found = CAP + 1;
  if (M2 > 1e-30f && M2 < 1e30f && S < 1e18f) {
    const float low = fmaxf(sqrtf(M2) - SUBPIX_MARGIN * S, 0.0f), thr = 0.999999f * low * low;
    if (threadIdx.x == 0) sh.redi[0] = 0;
    __syncthreads();
    if (most >= thr)
      for (int e = threadIdx.x; e < L * sp; e += PK_T) {
        float2 v[16];
        sixteenth(Tx + e % L, L, e / L, v);
#pragma unroll
        for (int b = 0; b < 16; b++)
          if (fmaf(v[b].x, v[b].x, v[b].y * v[b].y) >= thr) {
            const int at = atomicAdd(&sh.redi[0], 1);
            if (at < CAP) list[at] = (sp * b + e / L) * L + e % L;
          }
      }
    __syncthreads();
    found = sh.redi[0];
    __syncthreads();
  }
  auto take = [&](float2 acc, int e) {
    const float mag = sqrtf(fmaf(acc.x, acc.x, __fmul_rn(acc.y, acc.y)));
    if (mag > bv || (mag == bv && e < bi)) { bv = mag; bi = e; }
  };
  // m mod L (L need not be a power of two: 16 sp divides TWN)
  const bool pow2 = (L & (L - 1)) == 0;
  auto turn = [&](int m) {
    if (pow2) return m & (L - 1);
    m %= L;
    return m < 0 ? m + L : m;
  };
  // row fyi of the intermediate, and the plane from it, term by term
  auto row_term = [&](int fyi, int nx) {
    float2 acc = make_float2(0.0f, 0.0f);
    for (int fxi = 0; fxi < 16; fxi++) {
      const int fx = fxi - 8;
      acc = cadd(acc, cmul_rn(patchF[((fyi - 8) & 15) * 16 + (fx & 15)], Wl[turn(fx * nx)]));
    }
    return acc;
  };
  if (found <= CAP) {
    // a warp per candidate: 16 lanes' row terms, then the sum of them
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < found; i += PK_NW) {
      const int e = list[i], ny = e / L, nx = e - ny * L;
      const float2 t = row_term(lane & 15, nx);
      float2 acc = make_float2(0.0f, 0.0f);
      for (int fyi = 0; fyi < 16; fyi++) {
        const float2 r = make_float2(__shfl_sync(0xffffffffu, t.x, fyi), __shfl_sync(0xffffffffu, t.y, fyi));
        acc = cadd(acc, cmul_rn(r, Wl[turn((fyi - 8) * ny)]));
      }
      take(acc, e);
    }
  } else {  // a flat patch, or values out of the squares' range: every one
    for (int e = threadIdx.x; e < 16 * L; e += PK_T) Tx[e] = row_term(e / L, e % L);
    __syncthreads();
    for (int e = threadIdx.x; e < L * L; e += PK_T) {
      const int ny = e / L, nx = e - ny * L;
      float2 acc = make_float2(0.0f, 0.0f);
      for (int fyi = 0; fyi < 16; fyi++) acc = cadd(acc, cmul_rn(Tx[fyi * L + nx], Wl[turn((fyi - 8) * ny)]));
      take(acc, e);
    }
  }
  block_argmax(sh, bv, bi);
}

// One window per cluster of S CTAs (S = 1: a plain CTA).  Every CTA holds the
// whole window and filters its own rows; with S > 1 the statistics threads'
// sums stay in the CTA that made them and CTA 0 gathers them through
// distributed shared memory, steps the search and hands the next weights back:
// two cluster barriers per function value.
template <int S>
__global__ void __launch_bounds__(PK_T, 1) k_peaks(const float* __restrict__ cwin, int mS, zr_peak_params_t p,
                                               int pad, int vfloats, double xatol3, zr_peak_result_t* __restrict__ res,
                                               const float2* __restrict__ tw) {
  extern __shared__ __align__(16) float smf[];
  __shared__ PkShared sh;
  __shared__ float2 patchF[16 * 16];
  const int w = 2 * mS;
  const int w2 = w * w;
  const int win = blockIdx.x / S, rank = S > 1 ? blockIdx.x % S : 0;
  const int warp = threadIdx.x >> 5;
  float* C = smf;
  float* V = smf + ((w2 + 3) & ~3);
  const float* src = cwin + (size_t)win * w2;
  for (int e = threadIdx.x; e < w2; e += PK_T) C[e] = src[e];
  const PkRows lay = pk_rows<S>(w, pad, vfloats, rank);
  __syncthreads();
  const float origin = C[mS * w + mS];
  if (p.suppress_origin) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const int o = mS * w + mS;
      float s = C[o + w] + C[o + 1];
      s = s + C[o - w];
      s = s + C[o - w];
      s = s + C[o + w + 1];
      s = s + C[o - w + 1];
      s = s + C[o - w + 1];
      s = s + C[o - w - 1];
      C[o] = 0.125f * s;
    }
    __syncthreads();
  }
  // mean of the window: the centring constant of the one-pass variances
  // (any value near the mean serves; the statistics are exact sums around it)
  float ls = 0.0f;
  for (int e = threadIdx.x; e < w2; e += PK_T) ls += C[e];
  stats_warps(sh, ls, 0.0f, 0, 0.0f);
  __syncthreads();
  if (warp == 0) {
    const FiltStats t = stats_total(sh);
    if (threadIdx.x == 0) sh.bc[0] = t.s1;
  }
  __syncthreads();
  const float c = (float)(sh.bc[0] / (double)w2);

  // Statistics of one filter setting, in CTA 0 of the window: FiltStats on
  // thread 0 of warp 0 (and, MODE 1, the argmax on every thread).
  auto gather = [&](PkSums a, auto mode) {
    constexpr int MODE = decltype(mode)::value;
    if constexpr (S > 1) {
      cg::cluster_group cl = cg::this_cluster();
      const int nt = lay.nty * lay.cols;  // statistics threads of this CTA
      __syncthreads();                // F has been read
      float* Z = V;
      if ((int)threadIdx.x < nt) {
        Z[threadIdx.x] = a.s1;
        Z[nt + threadIdx.x] = a.s2;
        Z[2 * nt + threadIdx.x] = a.mx;
        if (MODE == 1) {
          Z[3 * nt + threadIdx.x] = a.bv;
          Z[4 * nt + threadIdx.x] = __int_as_float(a.bi);
          Z[5 * nt + threadIdx.x] = __int_as_float(a.cnt);
        }
      }
      cl.sync();
      if (rank != 0) return;
      const int t = threadIdx.x, ty = t / lay.cols, tx = t - ty * lay.cols;
      a = PkSums{0.0f, 0.0f, -INFINITY, -INFINITY, 0, 0x7fffffff};
      if (ty < lay.rb) {
        int o = 0;
        while ((o + 1) * lay.rb / S <= ty) o++;  // the CTA that owns ty
        const int t0 = o * lay.rb / S, n = ((o + 1) * lay.rb / S - t0) * lay.cols, i = (ty - t0) * lay.cols + tx;
        const float* R = cl.map_shared_rank(V, o);
        a.s1 = R[i];
        a.s2 = R[n + i];
        a.mx = R[2 * n + i];
        if (MODE == 1) {
          a.bv = R[3 * n + i];
          a.bi = __float_as_int(R[4 * n + i]);
          a.cnt = __float_as_int(R[5 * n + i]);
        }
      }
      if (MODE == 0) a.cnt = t == 0 ? w2 : 0;
    }
    stats_warps(sh, a.s1, a.s2, a.cnt, a.mx);
    if (MODE == 1) {
      block_argmax(sh, a.bv, a.bi);
      if (threadIdx.x == 0) {
        sh.bc[1] = a.bv;
        sh.bi[0] = a.bi;
      }
    }
    __syncthreads();
  };
  // CTA 0's weights and radii for every CTA of the window: the search's (ws, r
  // and go) or the last filter's (wy, wx, ry, rx).  They are kept apart because
  // CTA 0 writes the last filter's while the others still read the search's end.
  auto share = [&](auto search) {
    if constexpr (S > 1) {
      cg::cluster_group cl = cg::this_cluster();
      cl.sync();
      if (rank != 0) {
        const PkShared* lead = cl.map_shared_rank(&sh, 0);
        for (int i = threadIdx.x; i < 2 * PK_MAXR + 4; i += PK_T) {
          if constexpr (decltype(search)::value) {
            sh.ws[i] = lead->ws[i];
          } else {
            sh.wy[i] = lead->wy[i];
            sh.wx[i] = lead->wx[i];
          }
        }
        if (threadIdx.x == 0) {
          if constexpr (decltype(search)::value) {
            sh.r = lead->r;
            sh.go = lead->go;
          } else {
            sh.ry = lead->ry;
            sh.rx = lead->rx;
          }
        }
      }
      __syncthreads();
    } else {
      __syncthreads();
    }
  };
  constexpr int ROUNDS = S > 1 ? 2 : 1;
  using Mode0 = std::integral_constant<int, 0>;
  using Mode1 = std::integral_constant<int, 1>;

  double sig_opt = nan("");
  int nfev = 0;
  if (p.bmode == 1) {
    const double x0 = brent_first(p.opti_lo, p.opti_hi);
    if (rank == 0 && warp == 0) {
      const int r = gauss_weights(x0, sh.ws);
      if (threadIdx.x == 0) {
        sh.r = r;
        sh.go = 1;
      }
    }
    share(std::true_type());
    for (bool first = true; sh.go; first = false) {
      const int r = sh.r;
      const PkSums a = filter_rows<0, ROUNDS>(C, V, lay, mS, r, r, sh.ws, sh.ws, c, false);
      gather(a, Mode0());
      if (rank == 0 && warp == 0) {
        const FiltStats st = stats_total(sh);
        if (threadIdx.x == 0) {
          const double f = objective(st, c, (double)w2);
          if (first) brent_begin(sh, p.opti_lo, p.opti_hi, xatol3, x0, f);
          else brent_step(sh, xatol3, p.opti_maxiter, f);
        }
        __syncwarp();
        if (sh.go) {
          const int next = gauss_weights(sh.x, sh.ws);
          if (threadIdx.x == 0) sh.r = next;
        }
      }
      share(std::true_type());
    }
    sig_opt = sh.x;  // CTA 0
    nfev = sh.bi[1];
  }
  if (rank == 0 && warp == 0) {
    const double sy = p.bmode == 1 ? sig_opt : (p.bmode == 2 ? p.conv_sigma_y : 0.0);
    const double sx = p.bmode == 1 ? sig_opt : (p.bmode == 2 ? p.conv_sigma_x : 0.0);
    const int a = gauss_weights(sy, sh.wy);
    const int b = gauss_weights(sx, sh.wx);
    if (threadIdx.x == 0) {
      sh.ry = a;
      sh.rx = b;
    }
  }
  share(std::false_type());
  const int ry = sh.ry, rx = sh.rx;
  const PkSums sums = filter_rows<1, ROUNDS>(C, V, lay, mS, ry, rx, sh.wy, sh.wx, c, p.use_mask != 0);
  gather(sums, Mode1());
  if constexpr (S > 1) {
    cg::this_cluster().sync();  // CTA 0 has read the others' sums
    if (rank != 0) return;
  }
  FiltStats st{0.0, 0.0, 0.0f, 0};
  if (warp == 0) st = stats_total(sh);
  const float amax = (float)sh.bc[1];
  const int aidx = sh.bi[0];
  __syncthreads();
  const int cy = aidx / w, cx = aidx - (aidx / w) * w;
  const float cval = C[cy * w + cx];
  float corr = cval;
  int flags = 0;
  int sy = -1, sx = -1;  // sub-pixel argmax on the upsampled grid
  float bv = 0.0f;
  const int sp = p.sub_pix_reg;
  const int L = 16 * sp;
  if (sp > 1) {
    if (cy - PK_SUBR >= 0 && cy + PK_SUBR <= w && cx - PK_SUBR >= 0 && cx + PK_SUBR <= w) {
      // the 16 x 16 filtered patch around the peak, separably: the vertical
      // pass for its 16 rows over the 16 + 2 rx columns the horizontal taps
      // reach (reflected), then the horizontal pass; the same multiply-adds
      // in the same order as the full filter pass, so the same values
      __shared__ float patch[16 * 16];
      const int pw = 16 + 2 * rx;
      for (int e = threadIdx.x; e < 16 * pw; e += PK_T) {
        const int i = e / pw, j = e - (e / pw) * pw;
        const int y = cy - PK_SUBR + i;
        const int xx = reflect_idx(cx - PK_SUBR - rx + j, w);
        float acc = 0.0f;
        if (ry == 0) acc = C[y * w + xx];
        else
          for (int k = 0; k <= 2 * ry; k++) acc = fmaf(sh.wy[k], C[reflect_idx(y - ry + k, w) * w + xx], acc);
        V[e] = acc;
      }
      __syncthreads();
      for (int e = threadIdx.x; e < 256; e += PK_T) {
        const int i = e >> 4, j = e & 15;
        float f = 0.0f;
        if (rx == 0) f = V[i * pw + j];
        else
          for (int k = 0; k <= 2 * rx; k++) f = fmaf(sh.wx[k], V[i * pw + j + k], f);
        patch[e] = f;
      }
      __syncthreads();
      int bi;
      subpix_search(patch, sp, tw, (float2*)C, patchF, sh, bv, bi);  // the window is no longer needed
      sy = bi / L;
      sx = bi - (bi / L) * L;
    } else {
      flags |= 1;
    }
  }
  if (threadIdx.x == 0) {
    const double n = (double)st.n;
    const double m1 = st.s1 / n;
    const double var = st.s2 / n - m1 * m1;
    const double mean = (double)c + m1;
    const double peaksig = ((double)amax - mean) / sqrt(var > 0.0 ? var : 0.0);
    double shy = (double)cy - w / 2.0, shx = (double)cx - w / 2.0;
    if (sy >= 0) {
      const double ry0 = (double)cy - w / 2.0, rx0 = (double)cx - w / 2.0;
      shy = ry0 + ((double)sy - L / 2.0 + (ry0 > 0 ? 1.0 : (ry0 < 0 ? -1.0 : 0.0))) / sp;
      shx = rx0 + ((double)sx - L / 2.0 + (rx0 > 0 ? 1.0 : (rx0 < 0 ? -1.0 : 0.0))) / sp;
      corr = (float)((double)bv / 256.0);
    }
    zr_peak_result_t r;
    r.shift_y = shy;
    r.shift_x = shx;
    r.sigma = sig_opt;
    r.corr = corr;
    r.peaksig = (float)peaksig;
    r.origin = origin;
    r.cy = cy;
    r.cx = cx;
    r.flags = flags;
    r.nfev = nfev;
    res[win] = r;
  }
}

// ---------------------------------------------------------------------------
// Peak search on uncropped correlation planes (preShift, zorro.py:1089-1092
// and 1148-1168): each plane is the whole C x C correlation, ifftshifted.  The
// planes are too large for one CTA, so the steps are separate launches over a
// batch of planes, driven by the bounded Brent search that the host runs for
// every plane of the batch in lock step:
//   k_full_prepare   origin value, the suppressOrigin stencil, plane mean;
//   k_full_vert      axis-0 Gaussian pass (reflect), into a scratch plane;
//   k_full_horz      axis-1 pass, its value kept or not, per-CTA partial
//                    (sum (f - c), sum (f - c)^2, max f) of the statistic;
//   k_full_reduce    the partials in a fixed order (repeatable sums);
//   k_full_masked    the maxShift disc rolled by the plane's offset: masked
//                    argmax (first index on ties) and the partial sums over
//                    the disc for the peak significance;
//   k_full_finish    the reduction of those and the sub-pixel step.
// ``sel`` lists the planes a launch works on (grid z).

constexpr int FP_T = 256;   // threads of the filter and masked passes
constexpr int FP_TX = 32;   // columns per filter CTA
constexpr int FP_RY = 64;   // rows per filter CTA

__global__ void __launch_bounds__(1024) k_full_prepare(float* __restrict__ planes, int C, int suppress,
                                                       float* __restrict__ origin, float* __restrict__ mean) {
  __shared__ double red[32];
  float* P = planes + (size_t)blockIdx.x * C * C;
  const int o = (C / 2) * C + C / 2;
  if (threadIdx.x == 0) {
    origin[blockIdx.x] = P[o];
    if (suppress) {  // literal stencil of zorro.py:1082-1083 at the shifted origin
      float sm = P[o + C] + P[o + 1];
      sm = sm + P[o - C];
      sm = sm + P[o - C];
      sm = sm + P[o + C + 1];
      sm = sm + P[o - C + 1];
      sm = sm + P[o - C + 1];
      sm = sm + P[o - C - 1];
      P[o] = 0.125f * sm;
    }
  }
  __syncthreads();
  float ls = 0.0f;
  double ds = 0.0;
  int cnt = 0;
  for (long long e = threadIdx.x; e < (long long)C * C; e += blockDim.x) {
    ls += P[e];
    if (++cnt == 64) { ds += ls; ls = 0.0f; cnt = 0; }
  }
  ds += ls;
  for (int off = 16; off > 0; off >>= 1) ds += __shfl_down_sync(0xffffffffu, ds, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ds;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
    mean[blockIdx.x] = (float)(t / ((double)C * C));
  }
}

// T[y][x] = sum_k wy[k] P[reflect(y + k - r)][x], the taps in order
__global__ void __launch_bounds__(FP_T) k_full_vert(const float* __restrict__ planes, int C, const int* __restrict__ sel,
                                                  const float* __restrict__ wts, const int* __restrict__ rad,
                                                  float* __restrict__ tmp) {
  const int j = blockIdx.z, p = sel[j];
  const int r = rad[2 * p];
  const float* w = wts + (size_t)p * 2 * (2 * PK_MAXR + 1);
  const float* P = planes + (size_t)p * C * C;
  float* T = tmp + (size_t)j * C * C;
  const int x = blockIdx.x * FP_TX + (threadIdx.x & (FP_TX - 1));
  if (x >= C) return;
  for (int y = blockIdx.y * FP_RY + threadIdx.x / FP_TX; y < min(C, (int)(blockIdx.y + 1) * FP_RY);
       y += FP_T / FP_TX) {
    float acc;
    if (r == 0) {
      acc = P[(size_t)y * C + x] * w[0];
    } else {
      acc = 0.0f;
      for (int k = 0; k <= 2 * r; k++) acc = fmaf(w[k], __ldg(P + (size_t)reflect_idx(y + k - r, C) * C + x), acc);
    }
    T[(size_t)y * C + x] = acc;
  }
}

// F[y][x] = sum_k wx[k] T[y][reflect(x + k - r)]; F kept when ``out`` is set;
// per-CTA partials of sum (F - c), sum (F - c)^2 and max F
__global__ void __launch_bounds__(FP_T) k_full_horz(const float* __restrict__ tmp, int C, const int* __restrict__ sel,
                                                  const float* __restrict__ wts, const int* __restrict__ rad,
                                                  const float* __restrict__ mean, float* __restrict__ out,
                                                  double* __restrict__ part) {
  __shared__ double red[FP_T / 32][3];
  const int j = blockIdx.z, p = sel[j];
  const int r = rad[2 * p + 1];
  const float* w = wts + (size_t)p * 2 * (2 * PK_MAXR + 1) + (2 * PK_MAXR + 1);
  const float* T = tmp + (size_t)j * C * C;
  const float c = mean[p];
  const int x = blockIdx.x * FP_TX + (threadIdx.x & (FP_TX - 1));
  float s1 = 0.0f, s2 = 0.0f, mx = -INFINITY;
  if (x < C) {
    for (int y = blockIdx.y * FP_RY + threadIdx.x / FP_TX; y < min(C, (int)(blockIdx.y + 1) * FP_RY);
         y += FP_T / FP_TX) {
      const float* row = T + (size_t)y * C;
      float f;
      if (r == 0) {
        f = row[x] * w[0];
      } else {
        f = 0.0f;
        for (int k = 0; k <= 2 * r; k++) f = fmaf(w[k], __ldg(row + reflect_idx(x + k - r, C)), f);
      }
      if (out) out[(size_t)p * C * C + (size_t)y * C + x] = f;
      const float d = f - c;
      s1 += d;
      s2 = fmaf(d, d, s2);
      mx = fmaxf(mx, f);
    }
  }
  double a = s1, b = s2, m = mx;
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
    m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = a;
    red[threadIdx.x >> 5][1] = b;
    red[threadIdx.x >> 5][2] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0, tm = -INFINITY;
    for (int i = 0; i < FP_T / 32; i++) {
      ta += red[i][0];
      tb += red[i][1];
      tm = fmax(tm, red[i][2]);
    }
    double* q = part + ((size_t)p * gridDim.y * gridDim.x + (size_t)blockIdx.y * gridDim.x + blockIdx.x) * 3;
    q[0] = ta;
    q[1] = tb;
    q[2] = tm;
  }
}

// stats[p] = (sum, sum of squares, max) over the partials of plane p, in order
__global__ void k_full_reduce(const double* __restrict__ part, int nblk, const int* __restrict__ sel,
                              double* __restrict__ stats) {
  const int p = sel[blockIdx.x];
  if (threadIdx.x != 0) return;
  double a = 0.0, b = 0.0, m = -INFINITY;
  const double* q = part + (size_t)p * nblk * 3;
  for (int i = 0; i < nblk; i++) {
    a += q[3 * i];
    b += q[3 * i + 1];
    m = fmax(m, q[3 * i + 2]);
  }
  stats[3 * p] = a;
  stats[3 * p + 1] = b;
  stats[3 * p + 2] = m;
}

constexpr int FP_MBLK = 128;  // CTAs per plane of the masked pass

// The disc of radius mS about the plane centre, np.roll-ed by (ry, rx)
// (zorro.py:1150-1153): pixel (y, x) is in it when the unrolled pixel
// ((y - ry) mod C, (x - rx) mod C) lies within mS of (C/2, C/2).
__device__ __forceinline__ bool in_rolled_disc(int y, int x, int C, int mS, int ry, int rx) {
  int yy = (y - ry) % C, xx = (x - rx) % C;
  if (yy < 0) yy += C;
  if (xx < 0) xx += C;
  const long long dy = yy - C / 2, dx = xx - C / 2;
  return dy * dy + dx * dx < (long long)mS * mS;
}

// Per-CTA partials over its share of plane p: the argmax of F * disc (zeros
// outside the disc compete, first index on ties) and sum (F - c),
// sum (F - c)^2 and the count over the disc.
__global__ void __launch_bounds__(FP_T) k_full_masked(const float* __restrict__ filt, int C, const int* __restrict__ sel,
                                                    int mS, const int* __restrict__ rolls,
                                                    const float* __restrict__ mean, double* __restrict__ part) {
  __shared__ float rv[FP_T / 32];
  __shared__ int ri[FP_T / 32];
  __shared__ double rs[FP_T / 32][3];
  const int p = sel[blockIdx.z];
  const float* F = filt + (size_t)p * C * C;
  const float c = mean[p];
  const int ry = rolls[2 * p], rx = rolls[2 * p + 1];
  float bv = -INFINITY, s1 = 0.0f, s2 = 0.0f;
  int bi = 0x7fffffff, cnt = 0;
  const long long n = (long long)C * C;
  for (long long e = (long long)blockIdx.x * FP_T + threadIdx.x; e < n; e += (long long)gridDim.x * FP_T) {
    const int y = (int)(e / C), x = (int)(e - (long long)y * C);
    const float f = F[e];
    const bool in = in_rolled_disc(y, x, C, mS, ry, rx);
    const float mv = in ? f : 0.0f;
    if (mv > bv || (mv == bv && (int)e < bi)) { bv = mv; bi = (int)e; }
    if (in) {
      const float d = f - c;
      s1 += d;
      s2 = fmaf(d, d, s2);
      cnt++;
    }
  }
  double a = s1, b = s2, k = cnt;
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_down_sync(0xffffffffu, bv, off);
    const int oi = __shfl_down_sync(0xffffffffu, bi, off);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    a += __shfl_down_sync(0xffffffffu, a, off);
    b += __shfl_down_sync(0xffffffffu, b, off);
    k += __shfl_down_sync(0xffffffffu, k, off);
  }
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    rv[wid] = bv;
    ri[wid] = bi;
    rs[wid][0] = a;
    rs[wid][1] = b;
    rs[wid][2] = k;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < FP_T / 32; i++) {
      if (rv[i] > rv[0] || (rv[i] == rv[0] && ri[i] < ri[0])) { rv[0] = rv[i]; ri[0] = ri[i]; }
      rs[0][0] += rs[i][0];
      rs[0][1] += rs[i][1];
      rs[0][2] += rs[i][2];
    }
    double* q = part + ((size_t)p * gridDim.x + blockIdx.x) * 5;
    q[0] = rv[0];
    q[1] = ri[0];
    q[2] = rs[0][0];
    q[3] = rs[0][1];
    q[4] = rs[0][2];
  }
}

// One CTA per plane: the masked partials in order, the peak significance,
// then the sub-pixel step on the filtered plane (or the integer fallback at
// the plane's edge) as k_peaks does it.
__global__ void __launch_bounds__(PK_T, 1) k_full_finish(const float* __restrict__ planes,
                                                       const float* __restrict__ filt, int C,
                                                       const int* __restrict__ sel, const double* __restrict__ part,
                                                       const float* __restrict__ mean, const float* __restrict__ origin,
                                                       const double* __restrict__ sigma, const int* __restrict__ nfev,
                                                       int sp, zr_peak_result_t* __restrict__ res,
                                                       const float2* __restrict__ tw) {
  extern __shared__ float2 scratch[];
  __shared__ PkShared sh;
  __shared__ float2 patchF[16 * 16];
  __shared__ float patch[16 * 16];
  __shared__ double fin[4];
  __shared__ int fidx;
  const int p = sel[blockIdx.x];
  if (threadIdx.x == 0) {
    const double* q = part + (size_t)p * FP_MBLK * 5;
    double bv = q[0], s1 = q[2], s2 = q[3], cnt = q[4];
    int bi = (int)q[1];
    for (int i = 1; i < FP_MBLK; i++) {
      const double* r = q + 5 * i;
      if (r[0] > bv || (r[0] == bv && (int)r[1] < bi)) { bv = r[0]; bi = (int)r[1]; }
      s1 += r[2];
      s2 += r[3];
      cnt += r[4];
    }
    if (bi == 0x7fffffff) {  // a plane of NaN, all of it inside the disc
      bv = nan("");
      bi = 0;
    }
    const double m1 = s1 / cnt;
    const double var = s2 / cnt - m1 * m1;
    fin[0] = ((double)(float)bv - ((double)mean[p] + m1)) / sqrt(var > 0.0 ? var : 0.0);
    fin[1] = bv;
    fidx = bi;
  }
  __syncthreads();
  const int cy = fidx / C, cx = fidx - (fidx / C) * C;
  const float* P = planes + (size_t)p * C * C;
  const float* F = filt + (size_t)p * C * C;
  double shy = (double)cy - C / 2.0, shx = (double)cx - C / 2.0;
  float corr = P[(size_t)cy * C + cx];
  int flags = 0;
  if (sp > 1) {
    if (cy - PK_SUBR >= 0 && cy + PK_SUBR <= C && cx - PK_SUBR >= 0 && cx + PK_SUBR <= C) {
      for (int e = threadIdx.x; e < 256; e += PK_T)
        patch[e] = F[(size_t)(cy - PK_SUBR + (e >> 4)) * C + cx - PK_SUBR + (e & 15)];
      __syncthreads();
      const int L = 16 * sp;
      float bv;
      int bi;
      subpix_search(patch, sp, tw, scratch, patchF, sh, bv, bi);
      const int sy = bi / L, sx = bi - (bi / L) * L;
      const double ry0 = (double)cy - C / 2.0, rx0 = (double)cx - C / 2.0;
      shy = ry0 + ((double)sy - L / 2.0 + (ry0 > 0 ? 1.0 : (ry0 < 0 ? -1.0 : 0.0))) / sp;
      shx = rx0 + ((double)sx - L / 2.0 + (rx0 > 0 ? 1.0 : (rx0 < 0 ? -1.0 : 0.0))) / sp;
      corr = (float)((double)bv / 256.0);
    } else {
      flags |= 1;
    }
  }
  if (threadIdx.x == 0) {
    zr_peak_result_t r;
    r.shift_y = shy;
    r.shift_x = shx;
    r.sigma = sigma[p];
    r.corr = corr;
    r.peaksig = (float)fin[0];
    r.origin = origin[p];
    r.cy = cy;
    r.cx = cx;
    r.flags = flags;
    r.nfev = nfev[p];
    res[p] = r;
  }
}

constexpr int PK_SMS = 152;                    // SMs: one CTA each
constexpr size_t PK_SMEM = (227 - 9) * 1024;  // dynamic shared memory beside the static arrays

// Whether one run of rows of a window split over S CTAs fits V (at two
// horizontal units a thread).
template <int S>
static bool pk_splits(int w, int vp, int vfloats) {
  const int rb = pk_ty(w), len = (pk_quad(w) ? 2 : 1) * ((rb + S - 1) / S);
  const int nt = ((rb + S - 1) / S) * (pk_quad(w) ? w / 4 : 64);
  return rb >= S && pk_vrows(w, vp, 2, vfloats) >= len && 6 * nt <= vfloats;
}

template <int S>
static int launch_peaks(const float* cwin, int M, int mS, const zr_peak_params_t& p, int pad, int vfloats, size_t smem,
                        zr_peak_result_t* res, const float2* tw, cudaStream_t st) {
  ZR_TRY(cuda_check(cudaFuncSetAttribute(k_peaks<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_peaks attr"));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(M * S);
  cfg.blockDim = dim3(PK_T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = S > 1 ? 1 : 0;
  ZR_TRY(cuda_check(cudaLaunchKernelEx(&cfg, k_peaks<S>, cwin, mS, p, pad, vfloats, p.opti_xatol / 3.0,
                                       res, tw), "k_peaks launch"));
  return launched("k_peaks");
}

static int full_blocks(int C) { return ((C + FP_TX - 1) / FP_TX) * ((C + FP_RY - 1) / FP_RY); }

}  // namespace zr

using namespace zr;

extern "C" int zr_locate_peaks(const float* cwin, int M, int max_shift, const zr_peak_params_t* params,
                               zr_peak_result_t* results, void* stream) {
  if (!cwin || !params || !results) return set_error(ZR_EINVAL, "zr_locate_peaks: null argument");
  if (M <= 0) return ZR_OK;
  const int w = 2 * max_shift;
  if (max_shift < 8 || max_shift > 112)
    return set_error(ZR_ESIZE, "zr_locate_peaks: maxShift %d outside [8, 112]", max_shift);
  if (params->sub_pix_reg > 1 && (TWN % (16 * params->sub_pix_reg) != 0 || 16 * params->sub_pix_reg > 512))
    return set_error(ZR_ESIZE, "zr_locate_peaks: subPixReg %d must be at most 32 and divide 2^10 * 3^2 * 5", params->sub_pix_reg);
  if (params->bmode == 2 && (4.0 * params->conv_sigma_y + 0.5 > PK_MAXR || 4.0 * params->conv_sigma_x + 0.5 > PK_MAXR))
    return set_error(ZR_ESIZE, "zr_locate_peaks: conv sigma too large");
  if (params->bmode == 1 && 4.0 * params->opti_hi + 0.5 > PK_MAXR)
    return set_error(ZR_ESIZE, "zr_locate_peaks: opti sigma bound too large");
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  // shared memory: the window, then V (the filter blocks; also the vertical
  // pass of the 16 x 16 sub-pixel patch)
  // (every sigma of the bounded search lies between its bounds, in either order;
  // gauss_weights cuts radii off at PK_MAXR)
  double smax = params->bmode == 1 ? fmax(params->opti_lo, params->opti_hi) : 0.0;
  if (params->bmode == 2) smax = fmax(params->conv_sigma_y, params->conv_sigma_x);
  const int pad = ((int)fmin(4.0 * fmax(smax, 0.0) + 0.5, (double)PK_MAXR) + 3) & ~3;
  const size_t win = (((size_t)w * w + 3) & ~(size_t)3) * sizeof(float);
  const size_t sub = (size_t)17 * 16 * params->sub_pix_reg * sizeof(float2);
  const size_t base = params->sub_pix_reg > 1 && win < sub ? sub : win;  // the sub-pixel step's scratch takes the window
  const size_t vmin = (size_t)16 * (16 + 2 * PK_MAXR) * sizeof(float);
  size_t vbytes = PK_SMEM > base + vmin ? PK_SMEM - base : vmin;
  if (vbytes > (size_t)64 * 1024) vbytes = 64 * 1024;
  const int vfloats = (int)(vbytes / sizeof(float));
  cudaStream_t st = (cudaStream_t)stream;
  // Windows below 96 pixels, each a CTA: two cluster barriers a function value
  // take longer than the rows they share out (20 windows of 40 x 40 169 us, 193
  // in clusters of two, 191 of four; of 82 x 82 201, 208 and 201; of 96 x 96
  // 199, 197 and 181; of 100 x 100 208, 191 and 171).  So are unfiltered windows
  // of any size, and those of one given filter where they are more than a wave:
  // a second wave that starts as SMs fall free takes less than a second launch
  // (190 of 128 x 128 unfiltered 29 us against 33, with a filter and 16-fold
  // sub-pixels 68 against 94; 20 of 200 x 200 with a filter 43 in clusters, 66
  // without).  In the search, full waves of one CTA per window and SM, then what
  // is left with as many CTAs per window as fit the SMs.
  if (w < 96 || (params->bmode != 1 && (params->bmode != 2 || M > PK_SMS)))
    return launch_peaks<1>(cwin, M, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st);
  const int full = M / PK_SMS * PK_SMS, rest = M - full;
  if (full) ZR_TRY(launch_peaks<1>(cwin, full, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st));
  cwin += (size_t)full * w * w;
  results += full;
  const int vp = ((w + 7) & ~7) + 2 * pad + 12;
  if (rest == 0) return ZR_OK;
  // (clusters sit within a GPC: not 19 of 8 CTAs fit at a time)
  if (rest <= 8 && pk_splits<8>(w, vp, vfloats))
    return launch_peaks<8>(cwin, rest, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st);
  if (rest <= 32 && pk_splits<4>(w, vp, vfloats))
    return launch_peaks<4>(cwin, rest, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st);
  if (rest <= 72 && pk_splits<2>(w, vp, vfloats))
    return launch_peaks<2>(cwin, rest, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st);
  return launch_peaks<1>(cwin, rest, max_shift, *params, pad, vfloats, base + vbytes, results, tw, st);
}

extern "C" int zr_full_prepare(float* planes, int n, int C, int suppress_origin, float* origin, float* mean,
                               void* stream) {
  if (!planes || !origin || !mean) return set_error(ZR_EINVAL, "zr_full_prepare: null argument");
  if (n <= 0) return ZR_OK;
  if (C < 32 || C > 8192 || (C & 1)) return set_error(ZR_ESIZE, "zr_full_prepare: plane side %d", C);
  k_full_prepare<<<n, 1024, 0, (cudaStream_t)stream>>>(planes, C, suppress_origin, origin, mean);
  return launched("k_full_prepare");
}

extern "C" size_t zr_full_work_bytes(int n_planes, int C) {
  const size_t filt_part = (size_t)n_planes * full_blocks(C) * 3 * sizeof(double);
  const size_t mask_part = (size_t)n_planes * FP_MBLK * 5 * sizeof(double);
  return (size_t)n_planes * C * C * sizeof(float) + (filt_part > mask_part ? filt_part : mask_part);
}

extern "C" int zr_full_filter(const float* planes, int n_planes, int C, const int* sel, int n_sel,
                              const float* weights, const int* radius, const float* mean, float* filtered,
                              double* stats, void* work, size_t work_bytes, void* stream) {
  if (!planes || !sel || !weights || !radius || !mean || !stats || !work)
    return set_error(ZR_EINVAL, "zr_full_filter: null argument");
  if (n_sel <= 0) return ZR_OK;
  if (n_sel > n_planes || C < 32 || C > 8192) return set_error(ZR_EINVAL, "zr_full_filter: bad sizes");
  if (work_bytes < zr_full_work_bytes(n_planes, C))
    return set_error(ZR_EWORK, "zr_full_filter: work buffer %zu < %zu", work_bytes, zr_full_work_bytes(n_planes, C));
  cudaStream_t st = (cudaStream_t)stream;
  float* tmp = (float*)work;
  double* part = (double*)((char*)work + (size_t)n_planes * C * C * sizeof(float));
  const dim3 grid((C + FP_TX - 1) / FP_TX, (C + FP_RY - 1) / FP_RY, n_sel);
  k_full_vert<<<grid, FP_T, 0, st>>>(planes, C, sel, weights, radius, tmp);
  ZR_TRY(launched("k_full_vert"));
  k_full_horz<<<grid, FP_T, 0, st>>>(tmp, C, sel, weights, radius, mean, filtered, part);
  ZR_TRY(launched("k_full_horz"));
  k_full_reduce<<<n_sel, 32, 0, st>>>(part, full_blocks(C), sel, stats);
  return launched("k_full_reduce");
}

extern "C" int zr_full_peaks(const float* planes, const float* filtered, int n_planes, int C, const int* sel,
                             int n_sel, int max_shift, const int* rolls, const float* mean, const float* origin,
                             const double* sigma, const int* nfev, int sub_pix_reg, zr_peak_result_t* results,
                             void* work, size_t work_bytes, void* stream) {
  if (!planes || !filtered || !sel || !rolls || !mean || !origin || !sigma || !nfev || !results || !work)
    return set_error(ZR_EINVAL, "zr_full_peaks: null argument");
  if (n_sel <= 0) return ZR_OK;
  if (n_sel > n_planes || C < 32 || C > 8192 || max_shift <= 0) return set_error(ZR_EINVAL, "zr_full_peaks: bad sizes");
  if (sub_pix_reg > 1 && (TWN % (16 * sub_pix_reg) != 0 || 16 * sub_pix_reg > 512))
    return set_error(ZR_ESIZE, "zr_full_peaks: subPixReg %d must be at most 32 and divide 2^10 * 3^2 * 5", sub_pix_reg);
  if (work_bytes < zr_full_work_bytes(n_planes, C))
    return set_error(ZR_EWORK, "zr_full_peaks: work buffer %zu < %zu", work_bytes, zr_full_work_bytes(n_planes, C));
  const float2* tw = twiddles();
  if (!tw) return ZR_ECUDA;
  cudaStream_t st = (cudaStream_t)stream;
  double* part = (double*)((char*)work + (size_t)n_planes * C * C * sizeof(float));
  k_full_masked<<<dim3(FP_MBLK, 1, n_sel), FP_T, 0, st>>>(filtered, C, sel, max_shift, rolls, mean, part);
  ZR_TRY(launched("k_full_masked"));
  const size_t smem = sub_pix_reg > 1 ? (size_t)17 * 16 * sub_pix_reg * sizeof(float2) : 16;
  ZR_TRY(cuda_check(cudaFuncSetAttribute(k_full_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "k_full_finish attr"));
  k_full_finish<<<n_sel, PK_T, smem, st>>>(planes, filtered, C, sel, part, mean, origin, sigma, nfev, sub_pix_reg,
                                           results, tw);
  return launched("k_full_finish");
}
