// Internal: the decode-sized layer (decode.cu) and its workspace.
#pragma once
#include "common.cuh"

namespace fmoe {

constexpr int kDecodeTokens = 8;  // most tokens of a call: one n8 column block of mma.sync per expert

// Router inputs of a call that starts from logits (logits == NULL: topk_ids / topk_weights are given)
struct RouteArgs {
  const float* logits = nullptr;  // [T, E]
  const float* bias = nullptr;    // grouped: [E] or NULL
  int grouped = 0, renorm = 1, n_group = 1, topk_group = 1;
  // or slots in expert order (sorted position -> slot, rows per expert, weights in sorted order)
  const int32_t* slot_of = nullptr;
  const int32_t* hist = nullptr;
  const float* gate = nullptr;
  bool small_scratch = false;  // the caller's scratch does not hold a faster family's plan: the decode kernels wherever they can take the call
};

struct DecodePlan {
  int64_t off_plan, off_ids, off_weights, off_xq, off_xs, off_act, off_z, off_counters, total;
  int stages, smem, x_bytes, n_red, n_epi, tp, red_bytes;
};

// Whether the decode kernels take this call; fills the plan (offsets into the workspace) when they do.
bool plan_decode(const fmoe_fused_args& a, const RouteArgs& r, DecodePlan* plan);
int run_decode(const fmoe_fused_args& a, const RouteArgs& r, const DecodePlan& plan, uint8_t* ws, cudaStream_t st);

}  // namespace fmoe
