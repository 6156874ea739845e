// In-place mixed-radix FFTs in shared memory whose first pass reads its
// inputs from a loader and whose last pass hands its outputs over in
// registers.
//
// A length L = 16 R2 R3 (R3 = 1: two passes) is transformed by decimation in
// time: with n = (n1 R2 + n2) R3 + n3 and k = k1 + 16 k2 + 16 R2 k3,
//   pass 1  16-point DFT over n1 for every (n2, n3)               -> k1
//   pass 2  twiddle W_(16 R2)^(n2 k1), R2-point DFT over n2       -> k2
//   pass 3  twiddle W_L^(n3 (k1 + 16 k2)), R3-point DFT over n3   -> k3
// and each pass overwrites only what the same thread has read (digit d_i of
// the address holds n_i before pass i and k_i after it).  One barrier
// separates two passes and nothing passes through shared memory before the
// first or after the last one: two barriers and two exchanges a transform,
// where the Stockham form of fft_core.cuh, staged on both sides, takes six
// barriers and four.  These kernels are bound by shared-memory bandwidth and
// by barrier and issue latency at 16 warps an SM, so that is what counts.
// Measured against the Stockham form (microseconds): forward spectra of eight
// K2 frames 838 -> 640, spectra, terms and 190 pair windows of twenty 1024 x
// 1024 frames 673 -> 538, terms and 190 pair windows at crop 2048 1324 -> 1143.
//
// Element (d1, d2, d3) of a sequence sits at d1 S1 + d2 R3 + d3 with S1 odd
// and = 1 (mod 16) from 512 points on: the lanes of a half-warp (8-byte
// accesses) then hit 16 distinct bank pairs in every pass, when they run over
// consecutive (n2, n3) in pass 1, over n3 and k1 = q, q + R3, ... in pass 2,
// over k1 in pass 3, or over 4 (2) sequences at pitch 4 (8) mod 16 with 4 (8)
// consecutive indices each.
#pragma once
#include "fft_core.cuh"
#include "internal.h"

namespace zr {

// The lengths and their radices.  (Up to 6144 the registration's transforms;
// the others serve Fourier binning.)
constexpr int IP_LENGTHS = 21;
__host__ __device__ constexpr int ip_length(int i) {
  switch (i) {
    case 0: return 64;
    case 1: return 128;
    case 2: return 256;
    case 3: return 384;
    case 4: return 512;
    case 5: return 768;
    case 6: return 1024;
    case 7: return 1536;
    case 8: return 2048;
    case 9: return 3072;
    case 10: return 4096;
    case 11: return 5120;
    case 12: return 5760;
    case 13: return 6144;
    case 14: return 7680;
    case 15: return 8192;
    case 16: return 9216;
    case 17: return 10240;
    case 18: return 11520;
    case 19: return 12288;
    case 20: return 15360;
    case 21: return 16384;
    default: return 0;
  }
}
static_assert(ip_length(IP_LENGTHS) == 16384 && ip_length(IP_LENGTHS + 1) == 0, "IP_LENGTHS is the last index");
__host__ __device__ constexpr int ip_r2(int L) {
  switch (L) {
    case 64: return 4;
    case 384: case 768: return 6;
    case 128: case 512: case 1024: return 8;
    case 1536: case 3072: return 12;
    case 256: case 2048: case 4096: case 5120: return 16;
    case 5760: return 18;
    case 6144: case 7680: case 9216: case 11520: case 12288: return 24;
    case 8192: case 10240: case 15360: case 16384: return 32;
    default: return 0;
  }
}
__host__ __device__ constexpr int ip_r3(int L) { return L / (16 * ip_r2(L)); }

template <int L>
struct Ip {
  static constexpr int R2 = ip_r2(L), R3 = ip_r3(L);
  static_assert(R2 > 0 && 16 * R2 * R3 == L, "transform length not supported");
  static constexpr int A1 = L / 16;                    // butterflies of pass 1
  static constexpr int S1 = A1 + 1;                    // address stride of digit 1
  static constexpr int RL = R3 > 1 ? R3 : R2;          // radix of the last pass
  static constexpr int NS = L / RL;                    // its butterflies
};

// Pitch of a sequence (float2s) when NB of them share the CTA's buffer.
__host__ __device__ constexpr int ip_ld(int L, int NB) {
  return ((16 * (L / 16 + 1) + 15) & ~15) + (NB >= 4 ? 4 : (NB == 2 ? 8 : 0));
}

// Threads of a CTA that transforms NB sequences: 32 elements a thread; the
// 24-point butterflies of 6144-point transforms want one a thread.
__host__ __device__ constexpr int ip_threads(int L, int NB) { return L > 4096 ? 512 : fft_threads(L, NB); }

// Complex sums and differences as packed pairs: one issue slot instead of
// two, the same roundings and the same FP32 throughput.
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

template <int DIR>
__device__ __forceinline__ void ip_dft4(float2& x0, float2& x1, float2& x2, float2& x3) {
  const float2 t0 = padd(x0, x2), t1 = psub(x0, x2), t2 = padd(x1, x3), d = psub(x1, x3);
  x0 = padd(t0, t2);
  x2 = psub(t0, t2);
  x1 = make_float2(t1.x - DIR * d.y, t1.y + DIR * d.x);  // t1 + DIR i d
  x3 = make_float2(t1.x + DIR * d.y, t1.y - DIR * d.x);
}

// cos, sin of 2 pi m / n at compile time (Taylor series within a quadrant).
__host__ __device__ constexpr double ip_sin(int m, int n) {
  m %= n;
  if (2 * m > n) return -ip_sin(n - m, n);  // sin(2 pi - x) = -sin x
  if (4 * m > n) m = n - 2 * m;             // sin(pi - x) = sin x, with halves kept: x = pi m / n below
  else m = 2 * m;
  const double x = 3.14159265358979323846 * m / n;
  double t = x, s = x;
  for (int i = 1; i < 14; i++) {
    t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double ip_cos(int m, int n) { return ip_sin(4 * m + n, 4 * n); }

// v * exp(DIR 2 pi i M / N)
template <int DIR, int M, int N>
__device__ __forceinline__ float2 ip_rot(float2 v) {
  constexpr float c = (float)ip_cos(M, N), s = (float)ip_sin(M, N);
  if constexpr (M % N == 0) return v;
  else if constexpr (4 * (M % N) == N) return make_float2(-DIR * v.y, DIR * v.x);
  else return make_float2(v.x * c - DIR * v.y * s, v.y * c + DIR * v.x * s);
}

template <int R, int DIR>
__device__ __forceinline__ void ip_dft(float2* x);

// R = A B: A-point DFTs over n1 (n = B n1 + n2), twiddles W_R^(n2 k1), B-point
// DFTs over n2; output k = k1 + A k2.
template <int A, int B, int DIR, int K1, int N2>
__device__ __forceinline__ void ip_comp_twiddle(float2 (&y)[B][A]) {
  y[N2][K1] = ip_rot<DIR, K1 * N2, A * B>(y[N2][K1]);
  if constexpr (K1 + 1 < A) ip_comp_twiddle<A, B, DIR, K1 + 1, N2>(y);
  else if constexpr (N2 + 1 < B) ip_comp_twiddle<A, B, DIR, 1, N2 + 1>(y);
}
template <int A, int B, int DIR>
__device__ __forceinline__ void ip_dft_comp(float2* x) {
  float2 y[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < A; n1++) y[n2][n1] = x[B * n1 + n2];
    ip_dft<A, DIR>(y[n2]);
  }
  ip_comp_twiddle<A, B, DIR, 1, 1>(y);
#pragma unroll
  for (int k1 = 0; k1 < A; k1++) {
    float2 z[B];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) z[n2] = y[n2][k1];
    ip_dft<B, DIR>(z);
#pragma unroll
    for (int k2 = 0; k2 < B; k2++) x[k1 + A * k2] = z[k2];
  }
}

template <int R, int DIR>
__device__ __forceinline__ void ip_dft(float2* x) {
  if constexpr (R == 2) {
    const float2 a = x[0], b = x[1];
    x[0] = padd(a, b);
    x[1] = psub(a, b);
  } else if constexpr (R == 3) {
    const float s = 0.86602540378443864676f;
    const float2 a = x[0], bc = padd(x[1], x[2]), d = psub(x[1], x[2]);
    const float2 t = make_float2(a.x - 0.5f * bc.x, a.y - 0.5f * bc.y);
    x[0] = padd(a, bc);
    x[1] = make_float2(t.x - DIR * s * d.y, t.y + DIR * s * d.x);
    x[2] = make_float2(t.x + DIR * s * d.y, t.y - DIR * s * d.x);
  } else if constexpr (R == 4) {
    ip_dft4<DIR>(x[0], x[1], x[2], x[3]);
  } else if constexpr (R == 6) {
    ip_dft_comp<2, 3, DIR>(x);
  } else if constexpr (R == 8) {
    ip_dft_comp<4, 2, DIR>(x);
  } else if constexpr (R == 12) {
    ip_dft_comp<4, 3, DIR>(x);
  } else if constexpr (R == 16) {
    ip_dft_comp<4, 4, DIR>(x);
  } else if constexpr (R == 5) {
    constexpr float c1 = (float)ip_cos(1, 5), c2 = (float)ip_cos(2, 5), s1 = (float)ip_sin(1, 5), s2 = (float)ip_sin(2, 5);
    const float2 a = x[0], b1 = padd(x[1], x[4]), b2 = padd(x[2], x[3]), d1 = psub(x[1], x[4]), d2 = psub(x[2], x[3]);
    const float2 t1 = make_float2(a.x + c1 * b1.x + c2 * b2.x, a.y + c1 * b1.y + c2 * b2.y);
    const float2 t2 = make_float2(a.x + c2 * b1.x + c1 * b2.x, a.y + c2 * b1.y + c1 * b2.y);
    const float2 u1 = make_float2(s1 * d1.x + s2 * d2.x, s1 * d1.y + s2 * d2.y);
    const float2 u2 = make_float2(s2 * d1.x - s1 * d2.x, s2 * d1.y - s1 * d2.y);
    x[0] = padd(a, padd(b1, b2));
    x[1] = make_float2(t1.x - DIR * u1.y, t1.y + DIR * u1.x);
    x[4] = make_float2(t1.x + DIR * u1.y, t1.y - DIR * u1.x);
    x[2] = make_float2(t2.x - DIR * u2.y, t2.y + DIR * u2.x);
    x[3] = make_float2(t2.x + DIR * u2.y, t2.y - DIR * u2.x);
  } else if constexpr (R == 18) {
    ip_dft_comp<6, 3, DIR>(x);
  } else if constexpr (R == 20) {
    ip_dft_comp<4, 5, DIR>(x);
  } else if constexpr (R == 24) {
    ip_dft_comp<8, 3, DIR>(x);
  } else if constexpr (R == 30) {
    ip_dft_comp<6, 5, DIR>(x);
  } else {
    static_assert(R == 32, "radix not supported");
    ip_dft_comp<8, 4, DIR>(x);
  }
}

// Twiddles of the passes, in tables of their own after the strided ones: for
// every length, W_(16 R2)^(r k1) as [r - 1][k1] for pass 2 (r < R2) and
// W_L^(r k) as [slot][k] for the last pass, whose slots hold r = 1, 2, 3 and
// 4, 8, 12 ... below RL (the others are products of two of them).  Lanes with
// consecutive k then read consecutive entries for every r, where the strided
// table costs a lane a cache line of its own for the larger r (60 instead of
// 12 L1 wavefronts for a warp's 16-point butterflies).
__host__ __device__ constexpr int ip_rl(int L) { return ip_r3(L) > 1 ? ip_r3(L) : ip_r2(L); }
__host__ __device__ constexpr int ip_slots(int R) { return R < 4 ? R - 1 : 3 + (R - 1) / 4; }
__host__ __device__ constexpr int ip_slot_r(int slot) { return slot < 3 ? slot + 1 : 4 * (slot - 2); }
__host__ __device__ constexpr int ip_tw2_size(int L) { return ip_r3(L) > 1 ? 16 * (ip_r2(L) - 1) : 0; }
__host__ __device__ constexpr int ip_tw_size(int L) { return ip_tw2_size(L) + ip_slots(ip_rl(L)) * (L / ip_rl(L)); }
// Offset of length L's tables (past the last length: their total).
__host__ __device__ constexpr int ip_tw_off(int L) {
  int off = 0;
  for (int i = 0; i <= IP_LENGTHS && ip_length(i) != L; i++) off += ip_tw_size(ip_length(i));
  return off;
}
constexpr int IP_TW = ip_tw_off(0);

template <int DIR>
__device__ __forceinline__ float2 ip_ldtw(const float2* __restrict__ p) {
  float2 w = __ldg(p);
  if (DIR > 0) w.y = -w.y;
  return w;
}

// v[r] *= W_(16 R2)^(r k1) (exp(DIR 2 pi i / M)), r = 1 .. R2-1.
template <int L, int DIR>
__device__ __forceinline__ void ip_twiddle2(float2* v, int k1, const float2* __restrict__ twtab) {
  constexpr int BASE = TWN + TW_COMPACT + ip_tw_off(L);
#pragma unroll
  for (int r = 1; r < Ip<L>::R2; r++) v[r] = cmul(v[r], ip_ldtw<DIR>(twtab + BASE + (r - 1) * 16 + k1));
}

// v[r] *= W_L^(r k), r = 1 .. RL-1, k < NS.
template <int L, int DIR>
__device__ __forceinline__ void ip_twiddle_last(float2* v, int k, const float2* __restrict__ twtab) {
  constexpr int R = Ip<L>::RL, NS = Ip<L>::NS, BASE = TWN + TW_COMPACT + ip_tw_off(L) + ip_tw2_size(L);
  const float2* __restrict__ tw = twtab + BASE + k;
  const float2 w1 = ip_ldtw<DIR>(tw), w2 = ip_ldtw<DIR>(tw + NS), w3 = ip_ldtw<DIR>(tw + 2 * NS);
  v[1] = cmul(v[1], w1);
  v[2] = cmul(v[2], w2);
  v[3] = cmul(v[3], w3);
#pragma unroll
  for (int a = 4; a < R; a += 4) {
    const float2 wa = ip_ldtw<DIR>(tw + (2 + a / 4) * NS);
    v[a] = cmul(v[a], wa);
    if (a + 1 < R) v[a + 1] = cmul(v[a + 1], cmul(wa, w1));
    if (a + 2 < R) v[a + 2] = cmul(v[a + 2], cmul(wa, w2));
    if (a + 3 < R) v[a + 3] = cmul(v[a + 3], cmul(wa, w3));
  }
}

// The sequence and butterfly of a pass's work item e: sequences fastest (BF,
// for kernels whose global accesses gather a few elements of each sequence)
// or butterflies fastest.
template <int NB, int COUNT, bool BF>
__device__ __forceinline__ void ip_split(int e, int& b, int& u) {
  if (BF) {
    b = e % NB;
    u = e / NB;
  } else {
    b = e / COUNT;
    u = e - b * COUNT;
  }
}

// Pass 1: butterfly (n2, n3) = j of sequence b takes elements j + r L/16 from
// ``load(b, j, v)``, which fills v[r] for r < 16.  A thread loads all its
// butterflies before it computes any, unless ONE_BY_ONE (loaders that need
// the registers themselves).
template <int L, int NB, int T, int DIR, bool BF, bool ONE_BY_ONE = false, typename Load>
__device__ __forceinline__ void ip_pass1(float2* s, Load load) {
  using P = Ip<L>;
  constexpr int NBF = NB * P::A1, K = (NBF + T - 1) / T, LD = ip_ld(L, NB);
  float2 v[ONE_BY_ONE ? 1 : K][16];
  auto fetch = [&](int i) {
    const int e = threadIdx.x + i * T;
    if ((NBF % T) == 0 || e < NBF) {
      int b, j;
      ip_split<NB, P::A1, BF>(e, b, j);
      load(b, j, v[ONE_BY_ONE ? 0 : i]);
    }
  };
  if (!ONE_BY_ONE) {
#pragma unroll
    for (int i = 0; i < K; i++) fetch(i);
  }
  constexpr int UNROLL = ONE_BY_ONE ? 1 : K;
#pragma unroll UNROLL
  for (int i = 0; i < K; i++) {
    if (ONE_BY_ONE) fetch(i);
    const int e = threadIdx.x + i * T;
    if ((NBF % T) == 0 || e < NBF) {
      int b, j;
      ip_split<NB, P::A1, BF>(e, b, j);
      float2* w = v[ONE_BY_ONE ? 0 : i];
      ip_dft<16, DIR>(w);
#pragma unroll
      for (int r = 0; r < 16; r++) s[b * LD + j + r * P::S1] = w[r];
    }
  }
}

// Pass 1 with butterflies j and j + 1 (j even) of one sequence in a thread, so
// that the loader can read neighbouring elements in one access: ``load(b, j,
// odd, v0, v1)`` fills v0 with butterfly j + odd and v1 with j + 1 - odd.
// Every other eight lanes take the odd one first (odd = 1): each store of a
// half-warp then covers all banks.
template <int L, int NB, int T, int DIR, typename Load>
__device__ __forceinline__ void ip_pass1_pairs(float2* s, Load load) {
  using P = Ip<L>;
  constexpr int NU = NB * (P::A1 / 2), LD = ip_ld(L, NB);
  static_assert(P::A1 % 2 == 0, "whole pairs");
  const int odd = (threadIdx.x >> 3) & 1;
  for (int e = threadIdx.x; e < NU; e += T) {
    const int b = e / (P::A1 / 2), j = 2 * (e - b * (P::A1 / 2));
    float2 v0[16], v1[16];
    load(b, j, odd, v0, v1);
    float2* p = s + b * LD + j;
    ip_dft<16, DIR>(v0);
#pragma unroll
    for (int r = 0; r < 16; r++) p[odd + r * P::S1] = v0[r];
    ip_dft<16, DIR>(v1);
#pragma unroll
    for (int r = 0; r < 16; r++) p[1 - odd + r * P::S1] = v1[r];
  }
}

// Pass 2 of a three-pass length, in place (nothing for a two-pass length).
template <int L, int NB, int T, int DIR, bool BF>
__device__ __forceinline__ void ip_pass2(float2* s, const float2* __restrict__ tw) {
  using P = Ip<L>;
  if constexpr (P::R3 > 1) {
    constexpr int R = P::R2, R3 = P::R3;
    constexpr int NBF = NB * 16 * R3, K = (NBF + T - 1) / T, LD = ip_ld(L, NB);
    float2 v[K][R];
    auto at = [&](int e, int& k1) {
      int b, u;
      ip_split<NB, 16 * R3, BF>(e, b, u);
      const int n3 = u % R3, g = u / R3;
      // without BF a half-warp covers all n3 of k1 = q, q + R3, ...
      k1 = BF || R3 >= 16 ? g : (g % (16 / R3)) * R3 + g / (16 / R3);
      return s + b * LD + k1 * P::S1 + n3;
    };
#pragma unroll
    for (int i = 0; i < K; i++) {
      const int e = threadIdx.x + i * T;
      if ((NBF % T) == 0 || e < NBF) {
        int k1;
        const float2* p = at(e, k1);
#pragma unroll
        for (int r = 0; r < R; r++) v[i][r] = p[r * R3];
      }
    }
#pragma unroll
    for (int i = 0; i < K; i++) {
      const int e = threadIdx.x + i * T;
      if ((NBF % T) == 0 || e < NBF) {
        int k1;
        float2* p = at(e, k1);
        ip_twiddle2<L, DIR>(v[i], k1, tw);
        ip_dft<R, DIR>(v[i]);
#pragma unroll
        for (int r = 0; r < R; r++) p[r * R3] = v[i][r];
      }
    }
    __syncthreads();
  }
}

// Inputs of the last pass's butterfly k (< NS) of sequence b.
template <int L, int NB>
__device__ __forceinline__ void ip_last_load(const float2* s, int b, int k, float2* v) {
  using P = Ip<L>;
  const float2* p = s + b * ip_ld(L, NB) + (P::R3 > 1 ? (k & 15) * P::S1 + (k >> 4) * P::R3 : k * P::S1);
#pragma unroll
  for (int r = 0; r < P::RL; r++) v[r] = p[r];
}

// The last pass: ``out(b, k, v)`` receives outputs k + r NS of every
// butterfly k of every sequence b.
// (FENCE: a barrier between the loads and the outputs, for an ``out`` that
// writes to ``s``.)
template <int L, int NB, int T, int DIR, bool BF, bool FENCE = false, typename Out>
__device__ __forceinline__ void ip_last(const float2* s, const float2* __restrict__ tw, Out out) {
  using P = Ip<L>;
  constexpr int NBF = NB * P::NS, K = (NBF + T - 1) / T;
  float2 v[K][P::RL];
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int e = threadIdx.x + i * T;
    if ((NBF % T) == 0 || e < NBF) {
      int b, k;
      ip_split<NB, P::NS, BF>(e, b, k);
      ip_last_load<L, NB>(s, b, k, v[i]);
    }
  }
  if (FENCE) __syncthreads();
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int e = threadIdx.x + i * T;
    if ((NBF % T) == 0 || e < NBF) {
      int b, k;
      ip_split<NB, P::NS, BF>(e, b, k);
      ip_twiddle_last<L, DIR>(v[i], k, tw);
      ip_dft<P::RL, DIR>(v[i]);
      out(b, k, v[i]);
    }
  }
}

// Where element x of a transform sits after ip_last_inplace.
template <int L>
__device__ __forceinline__ int ip_at(int x) {
  using P = Ip<L>;
  const int k = x % P::NS, r = x / P::NS;
  return (P::R3 > 1 ? (k & 15) * P::S1 + (k >> 4) * P::R3 : k * P::S1) + r;
}

// The last pass with its outputs left in shared memory (ip_at).
template <int L, int NB, int T, int DIR>
__device__ __forceinline__ void ip_last_inplace(float2* s, const float2* __restrict__ tw) {
  ip_last<L, NB, T, DIR, false>(s, tw, [&](int b, int k, const float2* v) {
#pragma unroll
    for (int r = 0; r < Ip<L>::RL; r++) s[b * ip_ld(L, NB) + ip_at<L>(k) + r] = v[r];
  });
}

// The last pass with butterflies k and NS - k of one sequence in one thread
// (k = 0 with NS/2), sequences fastest, so that X[m] meets X[L - m] in
// registers: output r of butterfly k is X[k + r NS], and X[L - k - r NS] is
// output RL-1-r of butterfly NS - k (k = 0: output (RL - r) mod RL of
// butterfly 0).  ``pair(b, k0, X0, k1, X1)`` receives both butterflies.
template <int L, int NB, int T, int DIR, typename Pair>
__device__ __forceinline__ void ip_last_paired(const float2* s, const float2* __restrict__ tw, Pair pair) {
  using P = Ip<L>;
  constexpr int NU = NB * (P::NS / 2);
  for (int e = threadIdx.x; e < NU; e += T) {
    const int b = e % NB, u = e / NB;
    const int k0 = u, k1 = u == 0 ? P::NS / 2 : P::NS - u;
    float2 x0[P::RL], x1[P::RL];
    ip_last_load<L, NB>(s, b, k0, x0);
    ip_last_load<L, NB>(s, b, k1, x1);
    ip_twiddle_last<L, DIR>(x0, k0, tw);
    ip_twiddle_last<L, DIR>(x1, k1, tw);
    ip_dft<P::RL, DIR>(x0);
    ip_dft<P::RL, DIR>(x1);
    pair(b, k0, x0, k1, x1);
  }
}

// The circular convolution of length L with the sequence whose transform is
// ``hat`` (natural order), L times it: ``load(j, v)`` fills pass 1's inputs
// v[r] = x[j + r L/16], ``out(j, v)`` receives y[j + r L/16].  The inverse
// transform runs the passes backwards (decimation in frequency, twiddles after
// the butterflies), so its first butterflies take what the forward
// transform's last ones put out, element for element, with the product in
// registers between them: four exchanges through shared memory where two
// transforms with separate products take eight and the products two more.
// ``out`` may write to ``s``.
template <int L, int T, bool ONE_BY_ONE, typename Load, typename Out>
__device__ __forceinline__ void ip_convolve(float2* s, const float2* __restrict__ tw, const float2* __restrict__ hat,
                                            Load load, Out out) {
  using P = Ip<L>;
  static_assert(P::R3 > 1, "three passes");
  ip_pass1<L, 1, T, -1, false, ONE_BY_ONE>(s, [&](int, int j, float2* v) { load(j, v); });
  __syncthreads();
  ip_pass2<L, 1, T, -1, false>(s, tw);
  for (int k = threadIdx.x; k < P::NS; k += T) {
    float2 v[P::RL];
    float2* p = s + (k & 15) * P::S1 + (k >> 4) * P::R3;
#pragma unroll
    for (int r = 0; r < P::RL; r++) v[r] = p[r];
    ip_twiddle_last<L, -1>(v, k, tw);
    ip_dft<P::RL, -1>(v);
#pragma unroll
    for (int r = 0; r < P::RL; r++) v[r] = cmul(v[r], __ldg(hat + k + r * P::NS));
    ip_dft<P::RL, 1>(v);
    ip_twiddle_last<L, 1>(v, k, tw);
#pragma unroll
    for (int r = 0; r < P::RL; r++) p[r] = v[r];
  }
  __syncthreads();
  for (int u = threadIdx.x; u < 16 * P::R3; u += T) {
    const int n3 = u % P::R3, g = u / P::R3;
    const int k1 = P::R3 >= 16 ? g : (g % (16 / P::R3)) * P::R3 + g / (16 / P::R3);
    float2 v[P::R2];
    float2* p = s + k1 * P::S1 + n3;
#pragma unroll
    for (int r = 0; r < P::R2; r++) v[r] = p[r * P::R3];
    ip_dft<P::R2, 1>(v);
    ip_twiddle2<L, 1>(v, k1, tw);
#pragma unroll
    for (int r = 0; r < P::R2; r++) p[r * P::R3] = v[r];
  }
  __syncthreads();
  constexpr int K = (P::A1 + T - 1) / T;
  float2 v[K][16];
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int j = threadIdx.x + i * T;
    if (P::A1 % T == 0 || j < P::A1) {
#pragma unroll
      for (int r = 0; r < 16; r++) v[i][r] = s[j + r * P::S1];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int j = threadIdx.x + i * T;
    if (P::A1 % T == 0 || j < P::A1) {
      ip_dft<16, 1>(v[i]);
      out(j, v[i]);
    }
  }
}

// Output y of sequence b alone, |y| < NS (negative y: X[L + y]): the twiddled
// sum of butterfly y mod NS, without its other RL - 1 outputs.
template <int L, int NB, int DIR>
__device__ __forceinline__ float2 ip_last_one(const float2* s, int b, int y, const float2* __restrict__ tw) {
  using P = Ip<L>;
  float2 v[P::RL];
  ip_last_load<L, NB>(s, b, y < 0 ? y + P::NS : y, v);
  // W^(r y) for y < 0 is conj(W^(r |y|)): conjugate the inputs and the sum
  const float sg = y < 0 ? -1.0f : 1.0f;
#pragma unroll
  for (int r = 0; r < P::RL; r++) v[r].y *= sg;
  ip_twiddle_last<L, DIR>(v, y < 0 ? -y : y, tw);
  // (in the order of a radix-2 butterfly tree)
#pragma unroll
  for (int st = P::RL / 2; st > 0; st >>= 1)
#pragma unroll
    for (int r = 0; r < st; r++) v[r] = padd(v[r], v[r + st]);
  v[0].y *= sg;
  return v[0];
}

}  // namespace zr
