// Internal interface of the row kernels (rows.cu).
#pragma once
#include "common.cuh"

namespace fmoe {

// fmoe_gather_rows; without zero_padding the padding positions stay unwritten
int run_gather_rows(const void* x, int elem_bytes, int64_t rows_out, int64_t K, const int32_t* row_map, int map_div,
                    int64_t map_sentinel, const int32_t* num_rows_dev, void* out, bool zero_padding, cudaStream_t st);

// fmoe_quant_fp8_group128 / fmoe_quant_fp8_per_token, likewise
int run_quant_group128(const void* x, int in_dtype, int64_t rows_out, int64_t K, const int32_t* row_map, int map_div,
                       int64_t map_sentinel, const int32_t* num_rows_dev, void* q, float* scale, bool zero_padding,
                       cudaStream_t st);
int run_quant_per_token(const void* x, int in_dtype, int64_t rows_out, int64_t K, const int32_t* row_map, int map_div,
                        int64_t map_sentinel, const int32_t* num_rows_dev, void* q, float* scale, bool zero_padding,
                        cudaStream_t st);

#if defined(__CUDACC__)
// Scale of a group of 128 channels with this largest magnitude.
__device__ __forceinline__ float group_scale(float amax) { return __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f); }

// Eight values divided by the scale s (r = 1/s rounded) and rounded to e4m3; `finite`: none of the group is infinite.
__device__ __forceinline__ uint2 quant8(const float (&v)[8], float s, float r, bool finite) {
  uint32_t lo = 0, hi = 0;
  if (finite) {
    float q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = div_by_shared(v[i], s, r);
    // two values per conversion instruction (low byte = first value)
    auto pair = [](float a, float b) {
      return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    };
    lo = pair(q[0], q[1]) | (pair(q[2], q[3]) << 16);
    hi = pair(q[4], q[5]) | (pair(q[6], q[7]) << 16);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      lo |= (uint32_t)f32_to_e4m3_bits(__fdiv_rn(v[i], s)) << (8 * i);
      hi |= (uint32_t)f32_to_e4m3_bits(__fdiv_rn(v[4 + i], s)) << (8 * i);
    }
  }
  return make_uint2(lo, hi);
}
#endif

}  // namespace fmoe
