// Fourier binning: forward column pass.
#include "binning.cuh"

namespace zr {

// Frequencies -b0 .. b0 of column kx.
template <int Q, bool CHIRP>
__global__ void __launch_bounds__(bn_threads(Q), sm_minb(bn_threads(Q)))
    k_bin_cols(const float2* __restrict__ Ct, BnSide d, int b0, float2* __restrict__ Cc,
               const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const float2* col = Ct + (size_t)blockIdx.x * d.n;
  float2* o = Cc + (size_t)blockIdx.x * (2 * b0 + 1) + b0;
  bn_dft<Q, CHIRP>(sm, d, -b0, b0, tw, bn_each<Q>(d.n, [=](int j) { return __ldg(col + j); }), [&](int k, float2 X) { o[k] = X; });
}

int bn_cols(const float2* Ct, const BnSide& d, int Hb, int Kb, float2* Cc, const float2* tw, cudaStream_t st) {
  ZR_BN_DISPATCH(d, {
    const auto k = k_bin_cols<QQ, CC>;
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bn_smem<QQ>()),
                      "binning attr"));
    k<<<Kb, bn_threads(QQ), bn_smem<QQ>(), st>>>(Ct, d, Hb / 2, Cc, tw);
  })
  return launched("k_bin_cols");
}

}  // namespace zr
