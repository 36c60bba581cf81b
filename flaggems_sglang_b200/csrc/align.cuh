// Internal interface of moe_align (align.cu): the public outputs, and what the one-call layer asks for besides.
#pragma once
#include "common.cuh"

namespace fmoe {

struct AlignArgs {
  const int32_t* topk_ids = nullptr;
  int64_t numel = 0;
  int E = 0, block = 0;
  int32_t* sorted_ids = nullptr;
  int64_t sorted_cap = 0;
  int32_t* expert_ids = nullptr;
  int64_t expert_cap = 0;
  int32_t* num_post_pad = nullptr;
  void* workspace = nullptr;  // scratch of the multi-CTA variant (NULL: single CTA)
  int64_t workspace_bytes = 0;
  int32_t* table = nullptr;       // optional: expert table of the CTA-pair GEMMs (pair.cuh), for tiles of
  int token_tile = 256;           //   at most this many tokens
  int32_t* zero_words = nullptr;  // optional: counters of later kernels, set to zero
  int num_zero = 0;
  int32_t* slot_pos = nullptr;    // optional: [numel] position of every slot in the sorted order, -1 for dropped ids
  bool rows_only = false;         // padding positions and expert_ids are not read by anyone: they stay unwritten
  bool from_sorted = false;       // topk_ids is not read (run_align_sorted)
};
int run_align(const AlignArgs& a, cudaStream_t st);

// Slots that are already in expert order, and where their experts and weights go by slot.
struct SortedSlots {
  const int32_t* slot_of = nullptr;  // [numel] sorted position -> slot
  const int32_t* hist = nullptr;     // [E] rows per expert
  const float* gate = nullptr;       // [numel] weights in sorted order
  int32_t* ids = nullptr;            // [numel]
  float* weights = nullptr;          // [numel]
};
// The outputs of run_align from sorted slots; with sorted_ids == NULL only ids and weights.
int run_align_sorted(const AlignArgs& a, const SortedSlots& s, cudaStream_t st);

}  // namespace fmoe
