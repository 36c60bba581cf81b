// Internal: workspace plan and launcher of the one-call expert computation (fused.cu).
#pragma once
#include "common.cuh"
#include "decode.cuh"

namespace fmoe {

struct FusedPlan {
  int variant, block;
  int64_t numel, cap, nblk, max_blocks, total;
  // byte offsets into the workspace (-1: not used)
  int64_t off_sorted, off_expert, off_npp, off_align_ws, align_ws_bytes, off_xs, off_xs_scale, off_act, off_actq, off_actq_scale, off_z;
  int64_t off_split, split_bytes;  // tail-split scratch of the tcgen05 GEMMs
  bool use_decode;                  // the two decode kernels take the call (decode.cu); the fields above are then unused
  DecodePlan decode;
  int64_t off_route_ids, off_route_weights;  // calls from logits: where the router's results go (-1: not used)
  int64_t off_table, off_counters;  // expert table and tail-split counters of the CTA-pair GEMMs
  int64_t off_slot_pos;             // position of every slot in the sorted order
};

int pick_variant(int dtype, int64_t numel, int E, int64_t I, int64_t H, int forced, int* variant, int* block);
int plan_fused(const fmoe_fused_args& a, const RouteArgs& route, FusedPlan* plan);
// plan_fused for scratch of `limit` bytes: where the fastest family's plan is larger, that of the decode or the streaming kernels
// (no padded copies) if it fits.  The streaming ones only for calls of few rows per expert (pick_variant), or for `any_rows`: with
// many they would take many times as long, and a caller whose workspace is a little short is told so instead.  When none fits,
// the plan is the first one, and its total is above the limit.
int plan_within(const fmoe_fused_args& a, const RouteArgs& route, int64_t limit, bool any_rows, FusedPlan* plan);
// Enqueues the whole computation using `ws` (at least plan.total bytes, 256-byte aligned) as scratch.
int run_fused(const fmoe_fused_args& a, const RouteArgs& route, const FusedPlan& plan, uint8_t* ws, void* stream);

}  // namespace fmoe
