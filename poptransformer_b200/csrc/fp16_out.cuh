// Outputs of the products in fp16, four at a time.
#pragma once
#include "tile_math.cuh"

namespace pt {

// Four finished sums of an fp16 output, n .. n + 3 (n a multiple of four).
struct alignas(8) Half4 { __half v[4]; };
__device__ __forceinline__ Half4 load4(const __half *x, int n, int N, bool whole) {
  Half4 h;
  if (whole) *reinterpret_cast<uint2 *>(&h) = __ldcg(reinterpret_cast<const uint2 *>(x));
  else {
#pragma unroll
    for (int j = 0; j < 4; ++j) h.v[j] = n + j < N ? __ldcg(reinterpret_cast<const __half *>(x + j)) : __half(0);
  }
  return h;
}
__device__ __forceinline__ void store4(__half *o, const Half4 &h, int n, int N) {
  if (n + 4 <= N && ((uintptr_t)o & 7) == 0) *reinterpret_cast<uint2 *>(o) = *reinterpret_cast<const uint2 *>(&h);
  else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) o[j] = h.v[j];
  }
}

// (The branches are outside the elements: with them inside, a warp alone took 1100 cycles from the sums to the store.)
// GATED: PT_EPI_GATED_RESIDUAL is among them.
template <bool GATED> __device__ __forceinline__ Half4 finish4(int epilogue, const float4 &sum, const Half4 &res, const Half4 &bias, const Half4 &gate = Half4{}, bool halve = false) {
  __half2 y0 = __floats2half2_rn(sum.x, sum.y), y1 = __floats2half2_rn(sum.z, sum.w);
  const __half2 b0 = __halves2half2(bias.v[0], bias.v[1]), b1 = __halves2half2(bias.v[2], bias.v[3]), r0 = __halves2half2(res.v[0], res.v[1]), r1 = __halves2half2(res.v[2], res.v[3]);
  if (epilogue != PT_EPI_STORE) {
    if (epilogue == PT_EPI_RESIDUAL) {
      y0 = __hadd2_rn(r0, y0);
      y1 = __hadd2_rn(r1, y1);
    } else if (epilogue == PT_EPI_RELU2) {
      const __half2 zero = __float2half2_rn(0.f), p0 = __hgt2(y0, zero), p1 = __hgt2(y1, zero);      // (1 or 0; NaN gives 0)
      y0 = __halves2half2(__low2float(p0) != 0.f ? __low2half(y0) : __half(0), __high2float(p0) != 0.f ? __high2half(y0) : __half(0));
      y1 = __halves2half2(__low2float(p1) != 0.f ? __low2half(y1) : __half(0), __high2float(p1) != 0.f ? __high2half(y1) : __half(0));
      y0 = __hmul2_rn(y0, y0);
      y1 = __hmul2_rn(y1, y1);
    } else if (GATED && epilogue == PT_EPI_GATED_RESIDUAL) {
      y0 = __hadd2_rn(r0, __halves2half2(h_mul(sigmoid_h(gate.v[0]), __low2half(y0)), h_mul(sigmoid_h(gate.v[1]), __high2half(y0))));
      y1 = __hadd2_rn(r1, __halves2half2(h_mul(sigmoid_h(gate.v[2]), __low2half(y1)), h_mul(sigmoid_h(gate.v[3]), __high2half(y1))));
      if (halve) {
        y0 = __hmul2_rn(y0, __float2half2_rn(0.5f));
        y1 = __hmul2_rn(y1, __float2half2_rn(0.5f));
      }
    } else {
      y0 = __hadd2_rn(y0, b0);
      y1 = __hadd2_rn(y1, b1);
      if (epilogue == PT_EPI_BIAS_RESIDUAL) {
        y0 = __hadd2_rn(r0, y0);
        y1 = __hadd2_rn(r1, y1);
      } else if (epilogue == PT_EPI_BIAS_GELU) {
        y0 = __halves2half2(gelu_h(__low2half(y0)), gelu_h(__high2half(y0)));
        y1 = __halves2half2(gelu_h(__low2half(y1)), gelu_h(__high2half(y1)));
      }
    }
  }
  Half4 y;
  *reinterpret_cast<__half2 *>(&y.v[0]) = y0;
  *reinterpret_cast<__half2 *>(&y.v[2]) = y1;
  return y;
}

}  // namespace pt
