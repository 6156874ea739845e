// Fourier binning: forward row pass.
#include "binning.cuh"

namespace zr {

// Rows 2q and 2q+1 of the frame packed as x = a + i b; their half-plane rows
// kx in [0, Wb/2] written transposed, 16 bytes a frequency.
template <int Q, bool CHIRP>
__global__ void __launch_bounds__(bn_threads(Q), sm_minb(bn_threads(Q)))
    k_bin_rows(FrameSrc f, int n_frame, BnSide d, int b1, float2* __restrict__ Ct, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const int ya = 2 * blockIdx.x, H = f.H;
  const bool two = ya + 1 < H;
  // frequencies -b1 .. b1 in order
  bn_dft<Q, CHIRP, true>(
      sm, d, -b1, b1, tw,
      [&](int j, float2* v) {
        // a row's 16 pixels at a time, all their loads in flight together
        constexpr int FULL = CHIRP ? 0 : 16;
        float a[16], b[16];
        corrected16<Ip<Q>::A1, FULL>(f, n_frame, ya, j, f.W, a);
        if (two) corrected16<Ip<Q>::A1, FULL>(f, n_frame, ya + 1, j, f.W, b);
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = make_float2(a[r], two ? b[r] : 0.0f);
      },
      [&](int k, float2 X) { sm[k + b1] = X; });
  __syncthreads();
  // split: A_k = (Z_k + conj(Z_{-k})) / 2, B_k = (Z_k - conj(Z_{-k})) / (2i)
  for (int k = threadIdx.x; k <= b1; k += bn_threads(Q)) {
    const float2 z = sm[b1 + k], zm = sm[b1 - k];
    const float2 a = make_float2(0.5f * (z.x + zm.x), 0.5f * (z.y - zm.y));
    const float2 b = make_float2(0.5f * (z.y + zm.y), -0.5f * (z.x - zm.x));
    float2* o = Ct + (size_t)k * H + ya;
    if (two && (H & 1) == 0) {
      *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
    } else {
      o[0] = a;
      if (two) o[1] = b;
    }
  }
}

int bn_rows(const FrameSrc& f, int n, const BnSide& d, int Wb, float2* Ct, const float2* tw, cudaStream_t st) {
  ZR_BN_DISPATCH(d, {
    const auto k = k_bin_rows<QQ, CC>;
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bn_smem<QQ>()),
                      "binning attr"));
    k<<<(f.H + 1) / 2, bn_threads(QQ), bn_smem<QQ>(), st>>>(f, n, d, Wb / 2, Ct, tw);
  })
  return launched("k_bin_rows");
}

}  // namespace zr
