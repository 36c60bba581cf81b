// What the CTA-pair grouped GEMMs (gemm_pair.cu, gemm_pair_fold.cu) share: the table of experts, the tile order, the work
// units of a cluster and the TMA maps.
//
// Both kernels put the WEIGHTS on the M side of the tensor cores (256 weight rows per tile, 128 in each CTA of a pair)
// and the tokens on the N side.  N is any multiple of 16 up to the launch's token tile (64, 128 or 256), so an expert with
// 9 tokens costs a 16-column tile and one with 300 costs two of 160: no work is done for padding beyond 15 columns.  The
// rows between an expert's last token and the next multiple of the moe_align block are never touched.
#pragma once
#include "gemm.cuh"
#include "ptx_sm100.cuh"

namespace fmoe {

// Most tokens of a tile, by the rows an expert has on average.  A narrow tile leaves shared memory for a deeper ring of
// weights (what a launch needs whose time is the reading of weights); a wide one reads the weights from L2 less often.
// Experts well above the average are cut into several tiles either way.  bf16, layers with tiles of 128 / 256 in us, uniform
// routing: Mixtral rank, 83 rows 265 / 272, 115 rows 262 / 280, 130 rows 315 / 293; Qwen3 116 rows 263 / 269, 128 rows 304 / 287;
// with Zipf-1.2 routing: GPT-OSS 112 rows 372 / 346, Qwen3 94 rows 243 / 229.  The line of 88 costs uniform routing 2 to 7 % up to
// some 120 rows and saves skewed routing 6 to 7 %.  e4m3 multiplies a weight byte in half the time,
// so that the second reading is what counts (DeepSeek-V3, 64 rows on average: 128 tokens 2108 us, 256 tokens 1939 us).
inline int pick_token_tile(int64_t numel, int num_experts, bool e4m3) {
  const double rows = (double)numel / (double)(numel < num_experts ? (numel > 0 ? numel : 1) : num_experts);
  return rows <= 40.0 ? 64 : (rows <= 88.0 && !e4m3 ? 128 : 256);
}
// tail-split arrival counters of one launch: 8 per split tile, of which there are at most half as many as workers (<= 128); up to
// 126 workers the last word is free and counts the tickets (gemm_pair.cu)
constexpr int kSplitCounters = 512;

// int32 words of the expert table: first row [E], rows [E], exclusive prefix sum of the token tiles [E + 1]
__host__ __device__ constexpr int pair_table_words(int num_experts) { return 3 * num_experts + 1; }
__host__ __device__ constexpr int pair_table_bytes(int num_experts) { return (pair_table_words(num_experts) * 4 + 15) & ~15; }
// The e4m3 block-scale GEMMs (gemm_pair_fold.cu): experts with up to kNarrowRows rows go to the narrow kernel (one 64-token
// tile: 0.45 us per K block and tile, 0.36 with 16 rows), the others to the wide one (up to 128 tokens 0.50 us, 256 0.66 us).
// A call whose experts have few rows on average is left to the narrow kernel alone: the wide one would find next to nothing.
constexpr int kNarrowRows = 64;
inline bool fold_narrow_only(int64_t numel, int num_experts) {
  return numel <= 16 * (numel < num_experts ? numel : (int64_t)num_experts);
}

#if defined(__CUDACC__)
// Exclusive prefix sum over the experts' token tiles by one warp; rows[e] -> prefix[e], total in prefix[E].
__device__ __forceinline__ void pair_prefix_warp(const int32_t* rows, int32_t* prefix, int num_experts, int token_tile,
                                                 int lane) {
  int carry = 0;
  for (int base = 0; base < num_experts; base += 32) {
    const int e = base + lane;
    const int tiles = e < num_experts ? (rows[e] + token_tile - 1) / token_tile : 0;
    int incl = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (e < num_experts) prefix[e] = carry + incl - tiles;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) prefix[num_experts] = carry;
}

// All threads of the CTA fill `table` (shared memory): a copy of the one moe_align wrote, or, for callers of the plain
// C entry points, derived from the block tables (rows of an expert = up to the last real slot of its last block).
// Experts whose rows are outside [min_rows, max_rows] are left without tiles.  Ends with __syncthreads().
__device__ __forceinline__ void pair_build_table(int32_t* table, int num_experts, const int32_t* __restrict__ global_table,
                                                 const int32_t* __restrict__ expert_ids,
                                                 const int32_t* __restrict__ sorted_ids, int64_t numel, int block_rows,
                                                 int token_tile, int used_blocks, int min_rows = 0, int max_rows = 0x7fffffff) {
  int32_t* first = table;
  int32_t* rows = table + num_experts;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (global_table) {
    const bool all = min_rows <= 0 && max_rows == 0x7fffffff;
    for (int i = threadIdx.x; i < pair_table_words(num_experts); i += blockDim.x) {
      const int32_t v = __ldcg(global_table + i);  // possibly ahead of griddepcontrol.wait: not from L1
      table[i] = !all && i >= num_experts && i < 2 * num_experts && (v < min_rows || v > max_rows) ? 0 : v;
    }
    __syncthreads();
    if (all) return;
    if (warp == 0) pair_prefix_warp(rows, table + 2 * num_experts, num_experts, token_tile, lane);
    __syncthreads();
    return;
  }
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x) {
    first[e] = 0x7fffffff;
    rows[e] = 0;
  }
  __syncthreads();
  for (int b = threadIdx.x; b < used_blocks; b += blockDim.x) {
    const int e = expert_ids[b];
    if (e >= 0 && e < num_experts) {
      atomicMin(&first[e], b);
      atomicAdd(&rows[e], 1);
    }
  }
  __syncthreads();
  for (int e = warp; e < num_experts; e += blockDim.x >> 5) {
    const int b0 = first[e], nb = rows[e];
    __syncwarp();
    int last = 0;
    if (nb > 0) {
      const int64_t base = (int64_t)(b0 + nb - 1) * block_rows;
      for (int i = lane; i < block_rows; i += 32) {
        const int32_t s = sorted_ids[base + i];
        if (s >= 0 && s < numel) last = i + 1;
      }
      last = __reduce_max_sync(0xffffffffu, last);
    }
    if (lane == 0) {
      first[e] = nb > 0 ? b0 * block_rows : 0;
      const int r = nb > 0 ? (nb - 1) * block_rows + last : 0;
      rows[e] = r < min_rows || r > max_rows ? 0 : r;
    }
  }
  __syncthreads();
  if (warp == 0) pair_prefix_warp(rows, table + 2 * num_experts, num_experts, token_tile, lane);
  __syncthreads();
}

// One tile: `cols` real tokens (rows [row0, row0 + cols) of the sorted order) x weight tile `w_tile` of `expert`;
// n = cols rounded up to the 16 columns that an MMA of M = 256 steps by.
struct PairTile {
  int row0, cols, n, w_tile, expert;
  bool last;  // holds the expert's last token
};

// Tile order: expert by expert, inside an expert in groups of at most `group` token tiles, inside a group the token tile
// varies fastest: the tiles that run at the same time share weight rows through L2, and the group's token rows stay hot.
// Tokens per tile: the expert's in equal tiles, or, given a fixed number, as many per tile and the rest in the last.
// Int: int64_t, or int where the launch's tiles fit.
template <typename Int>
__device__ __forceinline__ PairTile pair_locate(Int tile, int w_tiles, int group, int num_experts, const int32_t* table,
                                                int fixed = 0) {
  const int32_t* prefix = table + 2 * num_experts;
  const int q = (int)(tile / w_tiles);
  int expert = 0, hi = num_experts - 1;  // last expert whose prefix is <= q (one with tiles, as q < prefix[E])
  while (expert < hi) {
    const int mid = (expert + hi + 1) >> 1;
    if (prefix[mid] <= q) expert = mid;
    else hi = mid - 1;
  }
  const int tiles = prefix[expert + 1] - prefix[expert];
  const int rows = table[num_experts + expert];
  const Int local = tile - (Int)prefix[expert] * w_tiles;
  const Int per_group = (Int)group * w_tiles;
  const int g = (int)(local / per_group), r = (int)(local % per_group);
  const int in_group = min(group, tiles - g * group);
  // where the last tile is a short one, the order changes from weight tile to weight tile: an even number of workers would
  // deal all short ones to half of them
  const int t = g * group + (fixed ? (r + r / in_group) % in_group : r % in_group);
  const int step = fixed ? fixed : (((rows + tiles - 1) / tiles) + 15) & ~15;
  PairTile tl;
  tl.w_tile = r / in_group;
  tl.row0 = table[expert] + t * step;
  tl.cols = min(step, rows - t * step);
  tl.n = (tl.cols + 15) & ~15;
  tl.expert = expert;
  tl.last = t == tiles - 1;
  return tl;
}

// ---- transposed stores ------------------------------------------------------------------------------
// A warp's strip of shared memory holds 16 tokens x (up to 32 channels + 8 of padding, so that neither the column stores
// nor the row loads conflict).
constexpr int kStripBytes = 16 * 80;

// 16 channels x 16 tokens in the fragment layout of tmem_ld_16x256b_x2, packed to bf16 (v[2 * token half + channel half]),
// into channels [ch, ch + 16) of a strip with `pitch` bytes per token.
__device__ __forceinline__ void strip_put16(uint8_t* strip, int pitch, int ch, int lane, const uint32_t (&v)[4]) {
  const int tok = (lane & 7) + (lane >> 4) * 8, c = ch + ((lane >> 3) & 1) * 8;
  ptx::stmatrix_x4_trans(ptx::smem_u32(strip + tok * pitch + c * 2), v[0], v[1], v[2], v[3]);
}
// 16 tokens x 16 channels of a strip (pitch 48) to consecutive rows; `rows` of them are real.
__device__ __forceinline__ void strip_store_sorted(const uint8_t* strip, int lane, __nv_bfloat16* out, int64_t n, int ch0,
                                                   int rows) {
  __syncwarp();
  const int u = lane >> 1, part = (lane & 1) * 8;
  const uint4 v = *reinterpret_cast<const uint4*>(strip + u * 48 + part * 2);
  if (u < rows && ch0 + part < n) *reinterpret_cast<uint4*>(out + u * n + ch0 + part) = v;
  __syncwarp();
}
// 16 tokens x 32 channels of a strip (pitch 80) to the rows of their slots; slot_a / slot_b: of tokens lane / 4 and
// 8 + lane / 4 (negative: none).
__device__ __forceinline__ void strip_store_slots(const uint8_t* strip, int lane, void* out, void* const* out_rows, int64_t n,
                                                  int ch0, int32_t slot_a, int32_t slot_b) {
  __syncwarp();
  const int part = (lane & 3) * 8;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 v = *reinterpret_cast<const uint4*>(strip + ((lane >> 2) + 8 * h) * 80 + part * 2);
    const int32_t slot = h ? slot_b : slot_a;
    if (slot >= 0 && ch0 + part < n) {
      __nv_bfloat16* row = out_rows ? reinterpret_cast<__nv_bfloat16*>(out_rows[slot])
                                    : reinterpret_cast<__nv_bfloat16*>(out) + (int64_t)slot * n;
      if (row) *reinterpret_cast<uint4*>(row + ch0 + part) = v;
    }
  }
  __syncwarp();
}
// gate/up GEMM through the plain C entry point: the rows between the expert's last token and the end of its 128-row block
// are zeros in this CTA's 64 channels (of elem_bytes each).  All `threads` epilogue threads.
__device__ __forceinline__ void zero_block_rows(const PairTile& tl, void* out, int64_t n, int ch, int elem_bytes, int thread,
                                                int threads) {
  const int from = tl.row0 + tl.cols, end = (from + 127) & ~127;  // blocks start at multiples of 128 rows
  const int per_row = 4 * elem_bytes;                              // 16-byte pieces
  for (int i = thread; i < (end - from) * per_row; i += threads) {
    const int64_t row = from + i / per_row, c = ch * elem_bytes + i % per_row * 16;
    if (c < n * elem_bytes) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(out) + row * n * elem_bytes + c) = make_uint4(0, 0, 0, 0);
  }
}
#endif

// Work units of one worker (a CTA pair).  Tiles are dealt round-robin (long launches of gemm_pair.cu: taken by ticket in the same
// order, a unit being that of worker ticket % workers in round ticket / workers); when the last round has work for at most half of
// the workers (they are bound by their own rate, so a part-filled round costs as much as a full one), each of its tiles
// is cut into S slices along K (S a power of two) that S neighbouring workers compute.  Every worker leaves its partial
// accumulator in global memory; whichever arrives last (counted per group of four epilogue warps) adds all S in slice order (a
// fixed order: results do not depend on timing) and runs the epilogue.  Nobody waits: workers may start in any order, and
// none needs another to be resident.  (Workers that wait for one another and finish a strip of the columns each need all of
// them resident; the times are the same: Mixtral rank, 333 tokens, 282 us per layer both ways, 287 against 281 without the
// split on another card.)
struct UnitPlan {
  int64_t total, rounds, left;
  int grid, b, S, k_steps;
  __host__ __device__ __forceinline__ void init(int64_t total_tiles, int k_steps_, int max_split, int grid_, int b_) {
    total = total_tiles;
    k_steps = k_steps_;
    grid = grid_;
    b = b_;
    S = 1;
    rounds = (total + grid - 1) / grid;
    left = total - (rounds - 1) * grid;
    if (total > 0 && max_split >= 2 && left * 2 <= grid) {
      int s = (int)(max_split < grid / left ? max_split : grid / left);
      s = s < k_steps / 8 ? s : k_steps / 8;
      while (s & (s - 1)) s &= s - 1;  // largest power of two below
      if (s >= 2) S = s;
    }
  }
  // unit `it` of this worker: tile, K steps [ks0, ks1), slice (always 0 for whole tiles); false past the last unit
  __host__ __device__ __forceinline__ bool get(int64_t it, int64_t* tile, int* ks0, int* ks1, int* slice) const {
    *ks0 = 0;
    *ks1 = k_steps;
    *slice = 0;
    if (S == 1 || it < rounds - 1) {
      *tile = b + it * grid;
      return *tile < total;
    }
    if (it > rounds - 1 || b >= left * S) return false;
    *tile = (rounds - 1) * grid + b / S;
    *slice = b % S;
    *ks0 = (int)((int64_t)k_steps * *slice / S);
    *ks1 = (int)((int64_t)k_steps * (*slice + 1) / S);
    return true;
  }
  __host__ __device__ __forceinline__ bool is_split(int64_t it) const { return S > 1 && it == rounds - 1; }
};

#if defined(__CUDACC__)
// A worker's units, worked out ahead of their use by one warp: 32 at a time, one per lane, in two batches of shared memory.
// Finding a unit is a search and seven divisions, which every role did for itself between two tiles while the tensor cores
// stood still.  Down GEMM of 128 experts, K = 768, 288 rows each: 162 -> 146 us, 512 rows 199 -> 184 us; DeepSeek-V3 layer of
// 128 tokens (narrow tiles, 56 and 16 K blocks) 1109 -> 1068 us.
constexpr int kListUnits = 32;
constexpr int kListBytes = 2 * kListUnits * 16;

struct PairUnit {
  PairTile tl;
  int slice, log2_s;  // slice of a tile that is cut into 2^log2_s along K
  int b;              // place in its round (UnitPlan)
  __device__ __forceinline__ int4 pack() const {
    return make_int4(tl.row0, tl.cols | (int)tl.last << 9 | log2_s << 10 | slice << 14, tl.w_tile, tl.expert | b << 16);
  }
  __device__ __forceinline__ void unpack(const int4& d) {
    tl.row0 = d.x;
    tl.cols = d.y & 511;
    tl.n = (tl.cols + 15) & ~15;
    tl.last = d.y >> 9 & 1;
    log2_s = d.y >> 10 & 15;
    slice = d.y >> 14;
    tl.w_tile = d.z;
    tl.expert = d.w & 0xffff;
    b = d.w >> 16;
  }
};

struct PairList {
  const int4* units;  // [2][kListUnits]; one without columns ends the list
  uint64_t* bars;     // full [2] (one arrival), empty [2] (one arrival per reading warp)
  int n = 0;          // units read so far
  __device__ __forceinline__ PairList(const void* units_, uint64_t* bars_) : units(reinterpret_cast<const int4*>(units_)), bars(bars_) {}
  static __device__ __forceinline__ void init_barriers(uint64_t* bars, int readers) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars[i], 1);
      ptx::mbar_init(&bars[2 + i], readers);
    }
  }
  // Next unit, for a role that one thread runs, or (WARP) a whole warp.  1: there is one, 0: the list has ended, -1: time-out.
  template <bool WARP>
  __device__ __forceinline__ int next(PairUnit* u) {
    const int batch = n / kListUnits, slot = batch & 1;
    if (n % kListUnits == 0) {
      if (WARP) __syncwarp();
      if (n && (!WARP || (threadIdx.x & 31) == 0)) ptx::mbar_arrive(&bars[2 + (slot ^ 1)]);
      bool ok = ptx::mbar_wait(&bars[slot], (batch >> 1) & 1);
      if (WARP) ok = __all_sync(0xffffffffu, ok);
      if (!ok) return -1;
    }
    u->unpack(units[slot * kListUnits + n % kListUnits]);
    ++n;
    return u->tl.cols != 0;
  }
  // A whole warp adds a batch of whole tiles: worker, worker + workers, .. below total.  1: there are more, 0: the list ends in it,
  // -1: time-out.
  static __device__ __forceinline__ int fill(int4* units, uint64_t* bars, int batch, int worker, int workers, int total, int w_tiles,
                                             int group, int num_experts, const int32_t* table, int fixed = 0) {
    const int slot = batch & 1, lane = threadIdx.x & 31;
    if (batch >= 2 && !__all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars[2 + slot], ((batch >> 1) & 1) ^ 1))) return -1;
    const int tile = worker + (batch * kListUnits + lane) * workers;
    int4 d = make_int4(0, 0, 0, 0);
    if (tile < total) {
      PairUnit u;
      u.tl = pair_locate(tile, w_tiles, group, num_experts, table, fixed);
      u.slice = u.log2_s = u.b = 0;
      d = u.pack();
    }
    units[slot * kListUnits + lane] = d;
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&bars[slot]);
    return __all_sync(0xffffffffu, tile < total);
  }
};
#endif

// TMA maps (gemm_pair.cu); 128-byte swizzle, zero fill
int encode_tensor_map(CUtensorMap* map, const void* base, int elem_bytes, int rank, const cuuint64_t* dims,
                      const cuuint64_t* strides, const cuuint32_t* box, bool weights, const char* what);
int pair_map_tokens(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int elem_bytes, int box_rows);
int pair_map_weights(CUtensorMap* map, const void* base, int64_t experts, int64_t n, int64_t k, int elem_bytes, bool gated,
                     bool interleaved = false);
int pair_map_weights_nmajor(CUtensorMap* map, const void* base, int64_t experts, int64_t k, int64_t w_rows);
int device_sm_count();

}  // namespace fmoe
