// Fourier binning: inverse row pass.
#include "binning.cuh"

namespace zr {

// Rows 2q and 2q+1 of the binned frame: the Hermitian rows of length Wb
// completed from kx in [0, Wb/2] and packed as a + i b, inverted.
template <int Q, bool CHIRP>
__global__ void __launch_bounds__(bn_threads(Q), sm_minb(bn_threads(Q)))
    k_bin_irows(const float2* __restrict__ Ci, BnSide d, int Hb, float* __restrict__ out,
                const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const int Wb = d.n, b1 = Wb / 2, i0 = 2 * blockIdx.x;
  float *oa = out + (size_t)i0 * Wb, *ob = oa + Wb;
  bn_dft<Q, CHIRP>(
      sm, d, 0, Wb - 1, tw,
      bn_each<Q>(Wb, [=](int m) {
        const int k = m <= b1 ? m : Wb - m;
        const float4 v = __ldg(reinterpret_cast<const float4*>(Ci + (size_t)k * Hb + i0));  // a_k, b_k
        float2 z;
        if (k == 0 || k == b1) z = make_float2(v.x, v.z);  // (their imaginary parts do not reach the real output)
        else if (m < b1) z = make_float2(v.x - v.w, v.y + v.z);
        else z = make_float2(v.x + v.w, -v.y + v.z);
        return cconj(z);
      }),
      [&](int x, float2 X) {
        oa[x] = X.x;
        ob[x] = -X.y;
      });
}

int bn_irows(const float2* Ci, const BnSide& d, int Hb, float* out, const float2* tw, cudaStream_t st) {
  ZR_BN_DISPATCH(d, {
    const auto k = k_bin_irows<QQ, CC>;
    ZR_TRY(cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bn_smem<QQ>()),
                      "binning attr"));
    k<<<Hb / 2, bn_threads(QQ), bn_smem<QQ>(), st>>>(Ci, d, Hb, out, tw);
  })
  return launched("k_bin_irows");
}

}  // namespace zr
