// Internal interface between the C-ABI entry points (api.cu) and the three
// grouped-GEMM kernel families.
#pragma once

#include "common.cuh"

namespace fmoe {

// e4m3 block-scale GEMMs: the two kernels share out the experts by their rows (gemm_pair_fold.cu); a caller that wants
// different outputs from them asks for one at a time.
enum class FoldKernel { kBoth, kNarrow, kWide };


// Arguments of one grouped GEMM: the public ones, and what only the one-call layer hands over (fused.cu).
struct GemmParams : fmoe_gemm_args {
  const int32_t* expert_table = nullptr;  // pair_table_words(E) words written by moe_align (see pair.cuh); NULL: derived
  bool behind_late_trigger = false;       // the launch before lets this one start only after its own wait (pdl_entry_late): the
                                          // table is complete then, and is read ahead of this kernel's wait
  int token_tile = 0;                     // the tile width that table was made for; 0: chosen by the launcher
  int32_t* split_counters = nullptr;      // zeroed arrival counters of the tail split; NULL: cleared by the launcher
  FoldKernel fold = FoldKernel::kBoth;
  bool fold_by_expert = false;            // kNarrow, gate/up: the output has kNarrowRows rows per expert, not one per position
  bool skip_padding = false;              // gate/up: rows between an expert's last row and its block's end stay unwritten
};

// gated = true : gemm1, w has 2*n rows per expert (gate rows then up rows), output
//                silu(gate)*up of width n, written at the sorted position p.
// gated = false: gemm2, w has n rows per expert, output written at row slot(p).
int gemm_simt(const GemmParams& p, bool gated, cudaStream_t st);
int gemm_stream(const GemmParams& p, bool gated, cudaStream_t st);
int gemm_pair(const GemmParams& p, bool gated, cudaStream_t st);
int gemm_pair_fold(const GemmParams& p, bool gated, cudaStream_t st);

// true when the variant can run these arguments (shape / alignment / dtype rules)
bool gemm_stream_supports(const GemmParams& p, bool gated);
bool gemm_pair_supports(const GemmParams& p, bool gated);
int64_t gemm_pair_split_workspace_bytes();
int tail_plan_unit(int64_t total_tiles, int k_steps, int max_split, int grid, int cta, int64_t it, int64_t* out);
// validates the arguments and launches the kernel family they ask for
int run_gemm(const GemmParams& p, bool gated, cudaStream_t st);
bool gemm_pair_fold_supports(const GemmParams& p, bool gated);

// Token tiles per group: the group's token rows should stay around 16 MB (hot in L2 across the weight tiles).
inline int pick_group_m(int64_t block_rows, int64_t k_bytes_per_row) {
  const int64_t per_block = block_rows * k_bytes_per_row;
  int64_t g = (16ll << 20) / (per_block > 0 ? per_block : 1);
  return (int)(g < 8 ? 8 : (g > 64 ? 64 : g));
}

// device status word written by bounded waits (gemm_pair.cu)
int read_and_clear_device_status(cudaStream_t st, int* status_out);

}  // namespace fmoe
