// Fourier binning: inverse column pass.
#include "binning.cuh"

namespace zr {

// Column kx of the cropped spectrum, made Hermitian, inverted: row i of it is
// frequency i (i < b0) or i - Hb.
template <int Q, bool CHIRP>
__global__ void __launch_bounds__(bn_threads(Q), sm_minb(bn_threads(Q)))
    k_bin_icols(const float2* __restrict__ Cc, BnSide d, int b1, float scale, float2* __restrict__ Ci,
                const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const int Hb = d.n, b0 = Hb / 2, kx = blockIdx.x;
  const float2* F = Cc + (size_t)kx * (Hb + 1) + b0;  // F[ky]
  float2* o = Ci + (size_t)kx * Hb;
  bn_dft<Q, CHIRP>(
      sm, d, 0, Hb - 1, tw,
      bn_each<Q>(Hb, [=](int i) {
        const int ky = i < b0 ? i : i - Hb;
        float2 v = __ldg(F + ky);
        if (kx < b1) {
          if (i == b0) {  // frequency -b0: averaged with +b0
            const float2 p = __ldg(F + b0);
            v = make_float2(0.5f * (v.x + p.x), 0.5f * (v.y + p.y));
          }
        } else if (i == b0) {  // the Nyquist column: F(ky, -b1) = conj(F(-ky, b1)) averaged with F(ky, b1)
          v = make_float2(__ldg(F + b0).x, 0.0f);
        } else {
          const float2 m = __ldg(F - ky);
          v = make_float2(0.5f * (v.x + m.x), 0.5f * (v.y - m.y));
        }
        return cconj(v);
      }),
      [&](int i, float2 X) { o[i] = make_float2(X.x * scale, -X.y * scale); });
}

int bn_icols(const float2* Cc, const BnSide& d, int Kb, int Wb, float scale, float2* Ci, const float2* tw,
             cudaStream_t st) {
  ZR_BN_DISPATCH(d, {
    const auto k = k_bin_icols<QQ, CC>;
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bn_smem<QQ>()),
                      "binning attr"));
    k<<<Kb, bn_threads(QQ), bn_smem<QQ>(), st>>>(Cc, d, Wb / 2, scale, Ci, tw);
  })
  return launched("k_bin_icols");
}

}  // namespace zr
