// moe_align_block_size: histogram -> scan -> stable scatter.
//
// Up to kOneLaunchSlots slots (and for any number without scratch) one launch does all of it: CTA b owns slots
// [1024 b, 1024 (b + 1)), one per thread, and counts ALL slots per expert, those before its own apart, so that no CTA waits
// for another.  Slots of an expert keep their ascending order: position = expert's start + slots before this CTA + slots in
// earlier warps + rank among the warp's equal ids (ballots).  Above that, three launches share the counting.
#include "align.cuh"
#include "ptx_sm100.cuh"

namespace fmoe {

__device__ int g_device_status_align = 0;  // this translation unit's status word; read by status_word_align()

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;

// Lanes of the warp whose id equals this lane's (ids below 2^bits; lanes without an id pass -1 and get the other such
// lanes).  One ballot per id bit: __match_any_sync took most of the 21 us of a single-CTA sort of 8192 slots.
__device__ __forceinline__ unsigned warp_peers(int id, int bits) {
  const bool on = id >= 0;
  unsigned peers = __ballot_sync(0xffffffffu, on);
  if (!on) peers = ~peers;
  for (int b = 0; b < bits; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (id >> b) & 1);
    peers &= ((id >> b) & 1) ? m : ~m;
  }
  return peers;
}
__host__ __device__ inline int id_bits(int E) {
  int b = 0;
  while ((1 << b) < E) ++b;
  return b;
}

// All NW warps of the CTA: exclusive scan of the padded row counts -> s_start[E + 1] and num_post_pad; with `table`, also the
// experts' first rows, rows and token tiles for the CTA-pair GEMMs (pair.cuh).  s_sum: [2 * NW].
template <int NW>
__device__ __forceinline__ void scan_experts(const int* s_total, int* s_start, int E, int block, int32_t* num_post_pad,
                                             int32_t* table, int token_tile, int* s_sum) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int carry = 0, tile_carry = 0;
  for (int base = 0; base < E; base += NW * 32) {
    const int e = base + tid;
    const int rows = (e < E) ? s_total[e] : 0;
    const int padded = ceil_div(rows, block) * block, tiles = ceil_div(rows, token_tile);
    int incl = padded, tile_incl = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off), w = __shfl_up_sync(0xffffffffu, tile_incl, off);
      if (lane >= off) {
        incl += v;
        tile_incl += w;
      }
    }
    if (lane == 31) {
      s_sum[warp] = incl;
      s_sum[NW + warp] = tile_incl;
    }
    __syncthreads();
    const int warps = min(NW, (E - base + 31) >> 5);  // the others' sums are zero
    int before = carry, tile_before = tile_carry;
    for (int w = 0; w < warps; ++w) {
      const int v = s_sum[w], u = s_sum[NW + w];
      if (w < warp) {
        before += v;
        tile_before += u;
      }
      carry += v;
      tile_carry += u;
    }
    if (e < E) {
      s_start[e] = before + incl - padded;
      if (table) {
        table[e] = before + incl - padded;
        table[E + e] = rows;
        table[2 * E + e] = tile_before + tile_incl - tiles;
      }
    }
    __syncthreads();  // s_sum is free again, s_start is complete
  }
  if (tid == 0) {
    s_start[E] = carry;
    if (num_post_pad) num_post_pad[0] = carry;
    if (table) table[3 * E] = tile_carry;
  }
  __syncthreads();
}

// What the block list holds besides the slots, shared out over the grid: block -> expert (-1 after the used blocks), and the
// sentinel in the padding of every expert and after the used blocks.
__device__ __forceinline__ void fill_padding(const int* s_total, const int* s_start, int E, int block, int numel,
                                             int32_t* sorted_ids, int sorted_cap, int32_t* expert_ids, int expert_cap) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, at = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * warps + (threadIdx.x >> 5); e < E; e += gridDim.x * warps) {
    for (int i = s_start[e] + s_total[e] + lane; i < min(s_start[e + 1], sorted_cap); i += 32) sorted_ids[i] = numel;
    for (int b = s_start[e] / block + lane; b < s_start[e + 1] / block && b < expert_cap; b += 32) expert_ids[b] = e;
  }
  for (int i = s_start[E] + at; i < sorted_cap; i += stride) sorted_ids[i] = numel;
  for (int b = s_start[E] / block + at; b < expert_cap; b += stride) expert_ids[b] = -1;
}

__global__ void __launch_bounds__(kThreads)
moe_align_kernel(const int32_t* __restrict__ topk_ids, int numel, int E, int block,
                 int32_t* __restrict__ sorted_ids, int sorted_cap, int32_t* __restrict__ expert_ids,
                 int expert_cap, int32_t* __restrict__ num_post_pad, int32_t* __restrict__ table, int token_tile,
                 int32_t* __restrict__ zero_words, int num_zero, int32_t* __restrict__ slot_pos, int rows_only) {
  pdl_entry();
  extern __shared__ int s_mem[];
  int* s_cnt = s_mem;                 // [kWarps][E] slots of this CTA's warps, then of the warps before
  int* s_before = s_mem + kWarps * E; // [E] slots of earlier CTAs
  int* s_total = s_before + E;        // [E]
  int* s_start = s_total + E;         // [E+1] padded start of each expert
  __shared__ int s_sum[2 * kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, bits = id_bits(E), first = blockIdx.x == 0;

  for (int i = tid; i < (kWarps + 2) * E; i += kThreads) s_mem[i] = 0;
  const int lo = blockIdx.x * kThreads, slot = lo + tid;
  int id = slot < numel ? topk_ids[slot] : -1;
  if (id < 0 || id >= E) id = -1;
  const unsigned peers = warp_peers(id, bits);
  const bool leader = id >= 0 && (__ffs(peers) - 1) == lane;
  __syncthreads();
  if (leader) s_cnt[warp * E + id] = __popc(peers);
  constexpr int kBatch = 8;
  const bool alone = gridDim.x == 1;  // this CTA's slots are all there are
  for (int base = tid; base < numel && !alone; base += kBatch * kThreads) {
    int v[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) v[i] = base + i * kThreads < numel ? topk_ids[base + i * kThreads] : -1;
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (v[i] >= 0 && v[i] < E) atomicAdd(base + i * kThreads < lo ? &s_before[v[i]] : &s_total[v[i]], 1);
  }
  __syncthreads();
  for (int e = tid; e < E; e += kThreads) {
    int run = s_before[e];
    s_total[e] += run;
#pragma unroll 8
    for (int w = 0; w < kWarps; ++w) {
      const int c = s_cnt[w * E + e];
      s_cnt[w * E + e] = run;
      run += c;
    }
    if (alone) s_total[e] = run;
  }
  __syncthreads();
  scan_experts<kWarps>(s_total, s_start, E, block, first ? num_post_pad : nullptr, first ? table : nullptr, token_tile, s_sum);

  if (slot < numel) {
    int pos = -1;
    if (id >= 0) {
      pos = s_start[id] + s_cnt[warp * E + id] + __popc(peers & ((1u << lane) - 1u));
      if (pos < sorted_cap) sorted_ids[pos] = slot;
    }
    if (slot_pos) slot_pos[slot] = pos;
  }
  for (int i = slot; i < num_zero; i += gridDim.x * kThreads) zero_words[i] = 0;
  if (!rows_only) fill_padding(s_total, s_start, E, block, numel, sorted_ids, sorted_cap, expert_ids, expert_cap);
}

// ---------------------------------------------------------------------------------------------
// Multi-CTA variant for large inputs: the slots are cut into chunks of kChunk, one CTA per chunk.
//   count   : per-chunk histogram -> cnt[chunk][E]; sentinel fill of sorted_token_ids
//   scan    : one CTA: exclusive scan over chunks per expert, padded starts, expert_ids, total
//   scatter : every CTA redoes its chunk's per-warp histogram and places its slots (stable)
// cnt and the experts' starts live in caller scratch ((chunks + 1) * E ints).
// ---------------------------------------------------------------------------------------------
constexpr int kChunk = 4096;
// Up to here every CTA counting all slots is faster than three dependent launches (8192 slots, 64 experts: one CTA 14.4 us).
constexpr int kOneLaunchSlots = 4 * kChunk;

__global__ void __launch_bounds__(kThreads)
align_count_kernel(const int32_t* __restrict__ topk_ids, int numel, int E, int32_t* __restrict__ sorted_ids,
                   int sorted_cap, int32_t* __restrict__ cnt, int rows_only) {
  pdl_entry();
  extern __shared__ int s_mem[];  // [E]
  const int tid = threadIdx.x;
  for (int e = tid; e < E; e += kThreads) s_mem[e] = 0;
  if (!rows_only)
    for (int64_t i = (int64_t)blockIdx.x * kThreads + tid; i < sorted_cap; i += (int64_t)gridDim.x * kThreads) sorted_ids[i] = numel;
  __syncthreads();
  const int lo = blockIdx.x * kChunk, hi = min(lo + kChunk, numel);
  int id[kChunk / kThreads];
#pragma unroll
  for (int i = 0; i < kChunk / kThreads; ++i) {
    const int s = lo + tid + i * kThreads;
    id[i] = s < hi ? topk_ids[s] : -1;
  }
#pragma unroll
  for (int i = 0; i < kChunk / kThreads; ++i)
    if (id[i] >= 0 && id[i] < E) atomicAdd(&s_mem[id[i]], 1);
  __syncthreads();
  for (int e = tid; e < E; e += kThreads) cnt[blockIdx.x * E + e] = s_mem[e];
}

__global__ void __launch_bounds__(kThreads)
align_scan_kernel(int chunks, int E, int block, int32_t* __restrict__ cnt, int32_t* __restrict__ starts,
                  int32_t* __restrict__ expert_ids,
                  int expert_cap, int32_t* __restrict__ num_post_pad, int32_t* __restrict__ table, int token_tile,
                  int32_t* __restrict__ zero_words, int num_zero, int rows_only) {
  pdl_entry();
  extern __shared__ int s_mem[];
  int* s_total = s_mem;      // [E]
  int* s_start = s_mem + E;  // [E+1]
  __shared__ int s_sum[2 * kWarps];
  const int tid = threadIdx.x;
  for (int i = tid; i < num_zero; i += kThreads) zero_words[i] = 0;
  for (int e = tid; e < E; e += kThreads) {
    int run = 0;
    for (int c0 = 0; c0 < chunks; c0 += 8) {
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = c0 + i < chunks ? cnt[(c0 + i) * E + e] : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c0 + i < chunks) cnt[(c0 + i) * E + e] = run;  // slots of e in earlier chunks
        run += v[i];
      }
    }
    s_total[e] = run;
  }
  __syncthreads();
  scan_experts<kWarps>(s_total, s_start, E, block, num_post_pad, table, token_tile, s_sum);
  const int used_blocks = s_start[E] / block;
  for (int e = tid; e < E; e += kThreads) starts[e] = s_start[e];  // first position of the expert, for the scatter
  if (rows_only) return;
  for (int e = tid; e < E; e += kThreads) {
    int b0 = s_start[e] / block, b1 = s_start[e + 1] / block;
    for (int b = b0; b < b1 && b < expert_cap; ++b) expert_ids[b] = e;
  }
  for (int b = used_blocks + tid; b < expert_cap; b += kThreads) expert_ids[b] = -1;
}

__global__ void __launch_bounds__(kThreads)
align_scatter_kernel(const int32_t* __restrict__ topk_ids, int numel, int E, const int32_t* __restrict__ cnt,
                     const int32_t* __restrict__ starts, int32_t* __restrict__ sorted_ids, int sorted_cap,
                     int32_t* __restrict__ slot_pos) {
  pdl_entry();
  extern __shared__ int s_mem[];  // [kWarps][E] per-warp counts -> running positions
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, bits = id_bits(E);
  for (int i = tid; i < kWarps * E; i += kThreads) s_mem[i] = 0;
  __syncthreads();
  constexpr int per_warp = kChunk / kWarps;  // 128 contiguous slots per warp
  const int lo = min(blockIdx.x * kChunk + warp * per_warp, numel), hi = min(lo + per_warp, numel);
  int id[per_warp / 32];
  unsigned peers[per_warp / 32];
#pragma unroll
  for (int i = 0; i < per_warp / 32; ++i) {
    const int s = lo + 32 * i + lane;
    id[i] = s < hi ? topk_ids[s] : -1;
    if (id[i] >= E) id[i] = -1;
  }
#pragma unroll
  for (int i = 0; i < per_warp / 32; ++i) {
    peers[i] = warp_peers(max(id[i], -1), bits);
    if (id[i] >= 0 && (__ffs(peers[i]) - 1) == lane) s_mem[warp * E + id[i]] += __popc(peers[i]);
    __syncwarp();
  }
  __syncthreads();
  for (int e = tid; e < E; e += kThreads) {
    int run = cnt[blockIdx.x * E + e] + starts[e];
#pragma unroll 8
    for (int w = 0; w < kWarps; ++w) {
      int c = s_mem[w * E + e];
      s_mem[w * E + e] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < per_warp / 32; ++i) {
    const int s = lo + 32 * i + lane;
    int pos = -1;
    if (id[i] >= 0) {
      pos = s_mem[warp * E + id[i]] + __popc(peers[i] & ((1u << lane) - 1u));
      if (pos < sorted_cap) sorted_ids[pos] = s;
    }
    if (slot_pos && s < hi) slot_pos[s] = pos;
    __syncwarp();
    if (id[i] >= 0 && (__ffs(peers[i]) - 1) == lane) s_mem[warp * E + id[i]] += __popc(peers[i]);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// The same tables from slots that the caller already holds in expert order (the reference operator's routing triple:
// sorted position -> slot, rows per expert, weights in sorted order): nothing is counted or sorted, every CTA scans the
// E row counts and copies its share of the positions to their padded places.  Also writes expert and weight by slot.
//
// The triple is the caller's memory and only the device sees it.  Rows past the last position are clipped, a position whose
// slot is outside [0, numel) is left out, and ids and slot_pos are -1 for a slot that no position names: no later kernel
// forms an address from a word that was not written in this call.  Both misuses are recorded for fmoe_check_device_status.
// Up to kSortedThreads slots one CTA sets them first, up to kClusterSlots a cluster, whose barrier stands between that and the
// first store of a position; above that a kernel before this one does it, because eight SMs take too long over the scattered
// stores.  64 experts of 1280 x 256, us per call, one CTA / cluster / two kernels: 8 slots 24.7 / 26.6 / -, 136 slots 45.1 /
// 45.2 / -, 2056 slots - / 52.9 / 51.3, 8192 slots - / 71.6 / 67.5, 32768 slots - / 176.2 / 155.5.
// ---------------------------------------------------------------------------------------------
constexpr int kSortedThreads = 256;
constexpr int kSortedCtas = 8;
constexpr int kClusterSlots = kSortedCtas * kSortedThreads;

__device__ __forceinline__ void report_triple(int code) { atomicCAS(&g_device_status_align, 0, code); }

__global__ void __launch_bounds__(kSortedThreads)
clear_slots_kernel(int numel, int32_t* __restrict__ ids, int32_t* __restrict__ slot_pos) {
  pdl_entry();
  for (int i = blockIdx.x * kSortedThreads + threadIdx.x; i < numel; i += gridDim.x * kSortedThreads) {
    ids[i] = -1;
    if (slot_pos) slot_pos[i] = -1;
  }
}

__global__ void __launch_bounds__(kSortedThreads)
align_sorted_kernel(const int32_t* __restrict__ slot_of, const int32_t* __restrict__ hist, const float* __restrict__ gate, int numel,
                    int E, int block, int32_t* __restrict__ sorted_ids, int sorted_cap, int32_t* __restrict__ expert_ids,
                    int expert_cap, int32_t* __restrict__ num_post_pad, int32_t* __restrict__ table, int token_tile,
                    int32_t* __restrict__ zero_words, int num_zero, int32_t* __restrict__ ids, float* __restrict__ weights,
                    int32_t* __restrict__ slot_pos, int rows_only, int clear) {
  pdl_entry();
  extern __shared__ int s_mem[];
  int* s_total = s_mem;            // [E]
  int* s_start = s_mem + E;        // [E+1] padded
  int* s_first = s_start + E + 1;  // [E+1] unpadded
  __shared__ int s_sum[2 * kSortedThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, block_id = blockIdx.x;
  const int stride = gridDim.x * kSortedThreads;
  if (clear) {
    for (int i = block_id * kSortedThreads + tid; i < numel; i += stride) {
      ids[i] = -1;
      if (slot_pos) slot_pos[i] = -1;
    }
  }
  for (int e = tid; e < E; e += kSortedThreads) s_total[e] = hist[e];
  __syncthreads();
  // Rows of every expert, and its first position: a prefix sum that stays at numel once it gets there (terms and sums are at
  // most numel < 2^30, so nothing overflows), so that the rows of all experts together are at most numel.
  if (warp == 0) {
    int carry = 0;
    bool over = false;
    for (int base = 0; base < E; base += 32) {
      const int e = base + lane, given = e < E ? s_total[e] : 0, v = min(max(given, 0), numel);
      int incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int w = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl = min(incl + w, numel);
      }
      incl = min(carry + incl, numel);
      int first = __shfl_up_sync(0xffffffffu, incl, 1);
      if (lane == 0) first = carry;
      if (e < E) {
        s_first[e] = first;
        s_total[e] = incl - first;
        over |= incl - first != given;
      }
      carry = __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_first[E] = carry;
    if (over && block_id == 0) report_triple(0xB01);
  }
  __syncthreads();
  scan_experts<kSortedThreads / 32>(s_total, s_start, E, block, block_id == 0 ? num_post_pad : nullptr,
                                    block_id == 0 ? table : nullptr, token_tile, s_sum);
  if (clear) ptx::cluster_sync_all();
  for (int p = block_id * kSortedThreads + tid; p < numel; p += stride) {
    const int slot = slot_of[p];
    const bool named = slot >= 0 && slot < numel;
    if (!named) report_triple(0xB00);
    if (p >= s_first[E]) continue;  // a histogram that does not cover every position: the rest belongs to no expert
    int lo = 0, hi = E - 1;         // last expert that starts at or before p
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_first[mid] <= p) lo = mid;
      else hi = mid - 1;
    }
    const int pos = s_start[lo] + p - s_first[lo];
    if (sorted_ids) sorted_ids[pos] = named ? slot : numel;  // pos < sorted_cap: at most numel rows (check_align)
    if (!named) continue;
    if (slot_pos) slot_pos[slot] = pos;
    ids[slot] = lo;
    weights[slot] = gate[p];
  }
  for (int i = block_id * kSortedThreads + tid; i < num_zero; i += stride) zero_words[i] = 0;
  if (sorted_ids && !rows_only) fill_padding(s_total, s_start, E, block, numel, sorted_ids, sorted_cap, expert_ids, expert_cap);
}

}  // namespace

namespace {
int check_align(const AlignArgs& a) {
  FMOE_REQUIRE(a.E >= 1 && a.E <= 1024, "moe_align_block_size: need 1 <= E <= 1024 (got %d)", a.E);
  FMOE_REQUIRE(a.block >= 1, "moe_align_block_size: block must be >= 1 (got %d)", a.block);
  FMOE_REQUIRE(a.numel >= 0 && a.numel < (1ll << 30), "moe_align_block_size: numel out of range");
  // worst case: every non-empty expert wastes block-1 positions
  const int64_t need = a.numel + (a.numel < a.E ? a.numel : (int64_t)a.E) * (a.block - 1);
  FMOE_REQUIRE(a.sorted_cap >= need, "moe_align_block_size: sorted_token_ids too small (%lld < %lld)",
               (long long)a.sorted_cap, (long long)need);
  FMOE_REQUIRE(a.sorted_cap < (1ll << 31), "moe_align_block_size: sorted_cap out of range");
  FMOE_REQUIRE(a.expert_cap >= ceil_div<int64_t>(a.sorted_cap, a.block),
               "moe_align_block_size: expert_ids too small (%lld < %lld)", (long long)a.expert_cap,
               (long long)ceil_div<int64_t>(a.sorted_cap, a.block));
  FMOE_REQUIRE(a.sorted_ids && a.expert_ids && a.num_post_pad && (a.topk_ids || a.numel == 0 || a.from_sorted),
               "moe_align_block_size: null pointer");
  return FMOE_OK;
}
}  // namespace

int run_align(const AlignArgs& a, cudaStream_t st) {
  int rc = check_align(a);
  if (rc) return rc;
  if (a.numel <= kOneLaunchSlots || !a.workspace) {
    const size_t smem = ((size_t)(kWarps + 3) * a.E + 1) * sizeof(int);
    if (smem > 48 * 1024)
      FMOE_CUDA_OK(cudaFuncSetAttribute(moe_align_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // a CTA per 1024 slots; with padding to fill, also one per 8192 positions
    const int64_t fill = a.rows_only ? 1 : std::min<int64_t>(16, ceil_div<int64_t>(a.sorted_cap, 8 * kThreads));
    const unsigned grid = (unsigned)std::max<int64_t>(std::max<int64_t>(1, fill), ceil_div<int64_t>(a.numel, kThreads));
    launch_pdl(moe_align_kernel, dim3(grid), dim3(kThreads), smem, st,
               a.topk_ids, (int)a.numel, a.E, a.block, a.sorted_ids, (int)a.sorted_cap, a.expert_ids, (int)a.expert_cap,
               a.num_post_pad, a.table, a.token_tile, a.zero_words, a.num_zero, a.slot_pos, (int)a.rows_only);
    return launch_status("moe_align_kernel");
  }
  FMOE_REQUIRE(a.workspace_bytes >= fmoe_moe_align_workspace_bytes(a.numel, a.E), "moe_align_block_size: workspace too small");
  const int chunks = (int)ceil_div<int64_t>(a.numel, kChunk);
  int32_t* cnt = static_cast<int32_t*>(a.workspace);
  int32_t* starts = cnt + (int64_t)chunks * a.E;
  launch_pdl(align_count_kernel, dim3(chunks), dim3(kThreads), a.E * sizeof(int), st, a.topk_ids, (int)a.numel, a.E, a.sorted_ids,
             (int)a.sorted_cap, cnt, (int)a.rows_only);
  rc = launch_status("align_count_kernel");
  if (rc) return rc;
  launch_pdl(align_scan_kernel, dim3(1), dim3(kThreads), (2 * a.E + 1) * sizeof(int), st, chunks, a.E, a.block, cnt, starts,
             a.expert_ids, (int)a.expert_cap, a.num_post_pad, a.table, a.token_tile, a.zero_words, a.num_zero, (int)a.rows_only);
  rc = launch_status("align_scan_kernel");
  if (rc) return rc;
  const size_t smem = (size_t)kWarps * a.E * sizeof(int);
  if (smem > 48 * 1024)
    FMOE_CUDA_OK(cudaFuncSetAttribute(align_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_pdl(align_scatter_kernel, dim3(chunks), dim3(kThreads), smem, st, a.topk_ids, (int)a.numel, a.E,
             (const int32_t*)cnt, (const int32_t*)starts, a.sorted_ids, (int)a.sorted_cap, a.slot_pos);
  return launch_status("align_scatter_kernel");
}

int run_align_sorted(const AlignArgs& a, const SortedSlots& s, cudaStream_t st) {
  FMOE_REQUIRE(a.E >= 1 && a.E <= 1024 && a.numel >= 1 && a.numel < (1ll << 30), "routing triple: bad E or slot count");
  FMOE_REQUIRE(s.slot_of && s.hist && s.gate && s.ids && s.weights, "routing triple: null pointer");
  if (a.sorted_ids) {
    const int rc = check_align(a);
    if (rc) return rc;
  }
  const bool clear = a.numel <= kClusterSlots;
  if (!clear) {
    launch_pdl(clear_slots_kernel, dim3(148), dim3(kSortedThreads), 0, st, (int)a.numel, s.ids, a.slot_pos);
    const int rc = launch_status("clear_slots_kernel");
    if (rc) return rc;
  }
  const int64_t items = std::max(a.numel, a.sorted_ids && !a.rows_only ? a.sorted_cap / 4 : 0);
  const unsigned cluster = !clear || a.numel <= kSortedThreads ? 1 : kSortedCtas;
  const unsigned grid = clear ? cluster : (unsigned)std::min<int64_t>(ceil_div<int64_t>(items, kSortedThreads), 148);
  launch_pdl_cluster(align_sorted_kernel, cluster, dim3(grid), dim3(kSortedThreads),
                     (3 * (size_t)a.E + 2) * sizeof(int), st, s.slot_of, s.hist, s.gate, (int)a.numel, a.E, a.block, a.sorted_ids,
                     (int)a.sorted_cap, a.expert_ids, (int)a.expert_cap, a.num_post_pad, a.table, a.token_tile, a.zero_words,
                     a.num_zero, s.ids, s.weights, a.slot_pos, (int)a.rows_only, (int)clear);
  return launch_status("align_sorted_kernel");
}

int status_word_align(int* out, bool clear) {
  int zero = 0;
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(out, g_device_status_align, sizeof(int)));
  if (clear && *out != 0) FMOE_CUDA_OK(cudaMemcpyToSymbol(g_device_status_align, &zero, sizeof(int)));
  return FMOE_OK;
}

}  // namespace fmoe

extern "C" int64_t fmoe_moe_align_workspace_bytes(int64_t numel, int E) {
  return (fmoe::ceil_div<int64_t>(numel > 0 ? numel : 1, fmoe::kChunk) + 1) * E * (int64_t)sizeof(int32_t);
}

extern "C" int fmoe_moe_align_block_size_ws(const int32_t* topk_ids, int64_t numel, int E, int block,
                                            int32_t* sorted_token_ids, int64_t sorted_cap, int32_t* expert_ids,
                                            int64_t expert_cap, int32_t* num_tokens_post_padded, void* workspace,
                                            int64_t workspace_bytes, void* stream) {
  fmoe::AlignArgs a;
  a.topk_ids = topk_ids;
  a.numel = numel;
  a.E = E;
  a.block = block;
  a.sorted_ids = sorted_token_ids;
  a.sorted_cap = sorted_cap;
  a.expert_ids = expert_ids;
  a.expert_cap = expert_cap;
  a.num_post_pad = num_tokens_post_padded;
  a.workspace = workspace;
  a.workspace_bytes = workspace_bytes;
  return fmoe::run_align(a, (cudaStream_t)stream);
}

extern "C" int fmoe_moe_align_block_size(const int32_t* topk_ids, int64_t numel, int E, int block,
                                         int32_t* sorted_token_ids, int64_t sorted_cap,
                                         int32_t* expert_ids, int64_t expert_cap,
                                         int32_t* num_tokens_post_padded, void* stream) {
  return fmoe_moe_align_block_size_ws(topk_ids, numel, E, block, sorted_token_ids, sorted_cap, expert_ids, expert_cap,
                                      num_tokens_post_padded, nullptr, 0, stream);
}
