// Internal interface of the row kernels (rows.cu).
#pragma once
#include "common.cuh"

namespace fmoe {

// fmoe_gather_rows; without zero_padding the padding positions stay unwritten
int run_gather_rows(const void* x, int elem_bytes, int64_t rows_out, int64_t K, const int32_t* row_map, int map_div,
                    int64_t map_sentinel, const int32_t* num_rows_dev, void* out, bool zero_padding, cudaStream_t st);

}  // namespace fmoe
