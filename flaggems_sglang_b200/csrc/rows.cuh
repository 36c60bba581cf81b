// Internal interface of the row kernels (rows.cu).
#pragma once
#include "common.cuh"

namespace fmoe {

// The layer's passes, by slot: slot_pos [T * k] is every slot's position in the sorted order (-1: none), as run_align
// writes it; padding positions are neither read nor written.
// token rows -> the positions of their k slots
int run_scatter_rows(const void* x, int elem_bytes, int64_t T, int k, int64_t K, const int32_t* slot_pos, void* out, cudaStream_t st);
// bf16 token rows -> e4m3 at the positions of their k slots; scales by token: [T, K/128], or [T] with per_row
int run_quant_scatter(const void* x, int64_t T, int k, int64_t K, const int32_t* slot_pos, bool per_row, void* q, float* scale,
                      cudaStream_t st);
// sorted bf16 rows -> e4m3 with one scale per row, in the same positions, scales by position
int run_quant_rows(const void* x, int64_t numel, int64_t K, const int32_t* slot_pos, void* q, float* scale, cudaStream_t st);
// sorted f32 rows -> e4m3 with a scale per 128 channels, likewise
int run_quant_slots(const float* x, int64_t numel, int64_t K, const int32_t* slot_pos, void* q, float* scale, cudaStream_t st);
// the same from max_rows f32 rows per expert to the experts' positions, only the experts with up to max_rows rows (table: pair.cuh): CTAs per expert, so that the other experts cost nothing
// (DeepSeek-V3, 4096 tokens, a third of the experts: 21 us against 105 us of looking at every slot)
int run_quant_experts(const float* x, int64_t numel, int64_t K, int num_experts, const int32_t* table, int max_rows, void* q,
                      float* scale, cudaStream_t st);

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
