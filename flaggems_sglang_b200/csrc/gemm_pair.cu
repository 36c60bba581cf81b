// Grouped GEMM on CTA pairs (cluster of 2, tcgen05 cta_group::2) for bf16 operands, and for e4m3 operands with one scale
// per token and one per output channel.
//
//   tile      : 256 weight rows (M, 128 in each CTA) x up to 64, 128 or 256 tokens of one expert (N, half loaded by each CTA)
//   K step    : 128 bytes per row (64 bf16 / 128 e4m3), one 128-byte swizzle atom; 4 MMAs per step
//   pipeline  : 192 KB ring of 6, 8 or 9 stages (16 KB of weights + 16, 8 or 4 KB of tokens) per CTA
//   TMEM      : 512 columns per CTA = two 128 x 256 fp32 accumulators, so the epilogue of a tile overlaps the next tile
//   warps     : 0-15 epilogue (TMEM lane quarter = warp % 4; the four of a quarter take 16-token chunks in turn),
//               16-17 TMA producers (each CTA its own weight rows and its own half of the tokens), 18 MMA issuer (CTA 0),
//               19 the worker's tiles (long launches: tickets, so that all workers stay near one another)
//
// Why pairs: with one CTA per 128 x 256 tile an MMA reads 12 KB of shared memory for every 8 KB here, and TMA writes as
// much; fill and operand reads of one SM together ran into its 128 bytes per clock.  Why weights on M: see pair.cuh.
//
// gate/up GEMM: a CTA's 128 weight rows are 64 gate and the matching 64 up rows, alternating in groups of 16, so that in
// the 16 x 256b read-out of TMEM a gate value and its up value land in the same thread; the activation is applied there
// and only [rows, I] is written.  Output is transposed 16 tokens at a time through a strip of shared memory private to the
// warp (stmatrix.trans), so that stores are 16 bytes of consecutive channels.
//
// Weights given as [E, K, N] (N contiguous) are read in place as an M-major operand, in 64-channel boxes: there the gate
// rows are lanes 0-63 and the up rows lanes 64-127, and the pairs meet through shared memory.
//
// Every mbarrier wait is bounded; on expiry the warp records a code in a device status word, leaves its loops, and the CTA
// frees its TMEM and returns.  The two cluster-wide barriers are reached by every thread on every path.  Every load has a
// single destination CTA.
#include "pair.cuh"

#include <cstdlib>
#include <mutex>

namespace fmoe {

__device__ int g_device_status = 0;  // 0 = fine; otherwise (role << 8 | site) of the first wait that gave up
// Optional wait-time profile (FMOE_TC_PROFILE=1): per CTA {tiles, mma wait acc, mma wait data, first producer's waits, epilogue wait,
// epilogue busy, second producer's waits}
__device__ long long g_wait_prof[256 * 8];

namespace {

constexpr int KBYTES = 128;
constexpr int W_BYTES = 128 * KBYTES;               // this CTA's weight rows of a stage
constexpr int RING_BYTES = 6 * 32 * 1024;           // stages of 16 KB of weights + half a token tile
constexpr int MAX_STAGES = 9;
constexpr int stage_bytes(int token_tile) { return W_BYTES + token_tile / 2 * KBYTES; }
constexpr int TMEM_COLS = 512;
constexpr int ACC_COLS = 256;
// Epilogue warps: 16 (4 per TMEM lane quarter), so that their TMEM, shuffle, shared-memory and store latencies overlap;
// with 8 a short main loop waited for them (7.3k cycles per tile against 6.1k of MMAs at K = 768).
constexpr int kEpiWarps = 16;
// TMA warps: they take the K steps in turn.  Waiting for a stage, arming it and issuing two to five copies takes one thread
// 430 to 500 cycles, and with one warp that was the pace of every tile whose MMAs need less.  SM cycles per K step, counted by the
// MMA warp, one / two warps: Mixtral gate/up with 192 tokens per tile 499 / 392 (their MMAs: 384), 256 tokens 515 / 513 (512);
// Qwen3 with 144 tokens 523 / 446.  A third warp changes nothing.  Qwen3, 128 experts of 288 rows: gate/up GEMM 270 -> 251 us.
constexpr int kProducers = 2;
constexpr int kThreads = (kEpiWarps + kProducers + 2) * 32;
constexpr int BOX_TOKENS = 32;                      // token rows per TMA box
constexpr int STRIP_BYTES = kStripBytes;             // per epilogue warp; also holds its 1 KB of the gate/up exchange
constexpr int BAR_BYTES = 768;
constexpr int kMaxTicketWorkers = (kSplitCounters - 1) / 8 * 2;  // the tail split leaves its last counter to the tickets
constexpr int smem_bytes(int num_experts) {
  return RING_BYTES + BAR_BYTES + kListBytes + kEpiWarps * STRIP_BYTES + pair_table_bytes(num_experts);
}
static_assert(smem_bytes(1024) <= 227 * 1024, "shared memory");

struct PairParams {
  const int32_t* sorted_token_ids;
  const int32_t* expert_ids;
  const int32_t* num_tokens_post_padded;
  const int32_t* expert_table;  // written by moe_align (NULL: derived from the block tables)
  bool early;                   // it is complete when the kernel starts
  const float* row_scale;
  const float* a_scale;   // F8: one scale per row of the sorted order, or per token (a_scale_gather)
  const float* w_scale;   // F8: [E, w_rows], one scale per output channel
  const float* bias;      // optional [E, w_rows]
  int32_t vec_step, vec_up;  // gate/up: entry of channel c in w_scale / bias is c * vec_step, its up entry vec_up further
  void* out;
  void* const* out_rows;  // down projection: optional per-slot row addresses (may be peer memory)
  float* split_partials;    // tail split: [workers][2 CTAs][128][256] f32 partial accumulators (NULL: no split)
  int32_t* split_counters;  // tail split: [tiles][2 CTAs][4 warp groups] arrivals, zero at launch
  int32_t* tickets;         // units taken beyond the workers' first ones, zero at launch (NULL: units are dealt round-robin)
  int64_t numel;
  int64_t n;              // gemm1: I, gemm2: H
  int64_t w_rows;         // rows of W per expert
  float act_alpha, act_limit;
  int32_t a_scale_gather;
  int32_t num_experts;
  int32_t k_steps;
  int32_t w_tiles;
  int32_t max_blocks;
  int32_t activation;
  int32_t group;
  int32_t profile;
  int32_t split_max;      // tail split: most K slices per tile (< 2: no split)
  int32_t top_k;
  int32_t a_rows;         // gather mode: rows of the input tensor (a row index >= a_rows reads zeros)
  int32_t token_tile;     // most tokens per tile
  int32_t stages, stage_bytes;
  int32_t zero_padding;   // gemm1: rows between an expert's last token and its block's end are written as zeros
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_device_status, 0, code); }

// Bounded wait whose verdict is uniform across the warp, so that the epilogue never diverges around __syncwarp().
__device__ __forceinline__ bool warp_wait_relaxed(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(bar, parity));
}

// Two epilogue warps (gate rows, up rows) meet.  Barriers 5-12; 1-4 are the groups of four, 0 is __syncthreads.
__device__ __forceinline__ void pair_of_warps_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(5 + pair) : "memory"); }

// Whether `pred` holds for any thread of the four epilogue warps (one of each TMEM lane quarter) that share barrier `bar`.
__device__ __forceinline__ bool any_of_four_warps(int bar, bool pred) {
  int v = pred;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %0, 0;\nbar.red.or.pred q, %1, 128, p;\nselp.s32 %0, 1, 0, q;\n}"
               : "+r"(v)
               : "r"(bar)
               : "memory");
  return v != 0;
}

// A worker's units in shared memory, two halves of kListUnits.  Dealt round-robin, each CTA's list warp works them out 32 at a
// time (as PairList).  Taken by ticket, CTA 0's does, one at a time and one unit ahead of the TMA warps, and hands them to the
// roles of both CTAs.
// Why tickets: workers with tiles of their own drift apart, by 108 us after 48 tiles of 27 us (Mixtral gate/up, 875 rows), since
// one that is behind finds its weights gone from L2 and falls further behind.  The four that share a weight tile were 37 us
// apart and read it from DRAM more than once; by ticket they are 2.4 us apart.  DRAM bytes read by that GEMM at 4096 tokens:
// 2.70 -> 1.95 GB, and 1.95 are its weights and rows.  (With one TMA warp, whose pace held the workers together, 1.99.  Dealt, it
// was 3.1 and 4.1 GB on other cards.)
struct PairFeed {
  const int4* units;  // [2 * kListUnits]; one without columns ends the work
  uint64_t* full;     // [2 * kListUnits] the unit, or (dealt) the 32 from it, are there
  uint32_t empty;     // [2] every reader has read a half: readers of this CTA, or (tickets) of both, in CTA 0
  uint64_t* ask;      // tickets, used in CTA 0: a TMA warp has begun a unit
  bool tickets;
  int n = 0;          // units read so far
  __device__ __forceinline__ PairFeed(const void* units_, uint64_t* bars, bool tickets_)
      : units(reinterpret_cast<const int4*>(units_)), full(bars), ask(bars + 2 * kListUnits + 2), tickets(tickets_) {
    empty = ptx::smem_u32(bars + 2 * kListUnits) & (tickets ? ~ptx::kPeerRankBit : ~0u);
  }
  __device__ __forceinline__ void init_barriers(int readers) {
    for (int i = 0; i < 2 * kListUnits; ++i) ptx::mbar_init(&full[i], 1);
    for (int i = 0; i < 2; ++i) ptx::mbar_init(full + 2 * kListUnits + i, readers);
    ptx::mbar_init(ask, 1);
  }
  __device__ __forceinline__ bool waits() const { return tickets || n % kListUnits == 0; }  // the next next() waits
  // Next unit, for a role that one thread runs, or (WARP) a whole warp.  1: there is one, 0: the work has ended, -1: time-out.
  template <bool WARP>
  __device__ __forceinline__ int next(PairUnit* u) {
    const int half = n / kListUnits, slot = n % (2 * kListUnits);
    if (n && n % kListUnits == 0) {
      if (WARP) __syncwarp();
      if (!WARP || (threadIdx.x & 31) == 0) ptx::mbar_arrive_cluster(empty + 8 * ((half & 1) ^ 1));
    }
    if (waits()) {
      bool ok = ptx::mbar_wait(&full[slot], (half >> 1) & 1);
      if (WARP) ok = __all_sync(0xffffffffu, ok);
      if (!ok) return -1;
    }
    u->unpack(units[slot]);
    ++n;
    return u->tl.cols != 0;
  }
  // The list warp, before it writes the first unit of a half: its readers have read what was there.
  __device__ __forceinline__ bool wait_half(int half) const {
    return half < 2 || __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(full + 2 * kListUnits + (half & 1), ((half >> 1) & 1) ^ 1));
  }
};

template <bool GATED, bool F8, bool EXTRA, bool WMN, bool GATHER>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
grouped_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_t, const __grid_constant__ CUtensorMap map_w,
                         const PairParams p) {
  constexpr int HALVES = kEpiWarps / 4;  // warps per lane quarter
  constexpr int kMmaWarp = kEpiWarps + kProducers;
  extern __shared__ __align__(1024) uint8_t smem[];  // aligned by declaration: every address below is a constant
  const int stages = p.stages, stage_size = p.stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + RING_BYTES);
  uint64_t* full_bar = bars;                    // [stages] used in CTA 0: the bytes of both CTAs' loads -> MMA
  uint64_t* empty_bar = bars + MAX_STAGES;          // [stages] per CTA: MMA -> this CTA's producer
  uint64_t* acc_full = bars + 2 * MAX_STAGES;       // [2] per CTA: MMA -> this CTA's epilogue
  uint64_t* acc_empty = bars + 2 * MAX_STAGES + 2;  // [2] used in CTA 0: both epilogues -> MMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 4);
  PairFeed units(smem + RING_BYTES + BAR_BYTES, bars + 2 * MAX_STAGES + 5, p.tickets != nullptr);
  uint8_t* strips = smem + RING_BYTES + BAR_BYTES + kListBytes;
  int32_t* table = reinterpret_cast<int32_t*>(strips + kEpiWarps * STRIP_BYTES);

  const int warp = ptx::uniform_warp_id(), lane = threadIdx.x & 31;
  const int rank = (int)ptx::cluster_ctarank();
  const int worker = blockIdx.x >> 1, workers = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);   // CTA 0's producer arms it with the bytes of both CTAs
      ptx::mbar_init(&empty_bar[s], 1);  // one tcgen05.commit
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&acc_full[a], 1);
      ptx::mbar_init(&acc_empty[a], 2 * kEpiWarps);  // one arrival per epilogue warp of both CTAs
    }
    units.init_barriers(units.tickets ? 2 * (kEpiWarps + kProducers) + 1 : kEpiWarps + kProducers + (rank == 0));
    ptx::fence_barrier_init();
  }
  if (warp == kEpiWarps && lane == 0) {
    ptx::prefetch_tensormap(&map_t);
    ptx::prefetch_tensormap(&map_w);
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  // Everything above is independent of the kernels before this one on the stream.  Behind a late trigger a given table is
  // complete by now (see pdl_entry_late): only the rows and what the epilogue reads and writes wait for the kernel before.
  const bool early = p.early;
  if (!early) pdl_wait();
  const int used_blocks = p.expert_table ? 0 : min((int)(*p.num_tokens_post_padded / 128), p.max_blocks);
  pair_build_table(table, p.num_experts, p.expert_table, p.expert_ids, p.sorted_token_ids, p.numel, 128,
                   p.token_tile, used_blocks);
  ptx::cluster_sync_all();  // the other CTA's barriers exist before anything is signalled across
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int k_steps = p.k_steps;
  PairUnit unit;
  const PairTile& tl = unit.tl;
  auto first_step = [&](int slice) { return (int)((int64_t)k_steps * slice >> unit.log2_s); };  // of a slice of this unit's tile

  if (warp >= kEpiWarps && warp < kMmaWarp) {
    // ---------------- TMA producers (both CTAs): K steps me, me + kProducers, .. of all the worker's tiles ----------------
    if (ptx::elect_one()) {
      const int me = warp - kEpiWarps;
      int stage = me, mine = me;  // mine: this warp's next K step, counted from the tile's first
      uint32_t phase = 0;
      int last_stage = -1;
      uint32_t last_phase = 0;
      auto advance = [&]() {
        last_stage = stage;
        last_phase = phase;
        stage += kProducers;
        if (stage >= stages) {
          stage -= stages;
          phase ^= 1;
        }
      };
      bool alive = true;
      long long prof_p = 0;
      const uint32_t ring = ptx::smem_u32(smem), bar_full0 = ptx::smem_u32(full_bar) & ~ptx::kPeerRankBit;
      for (bool first = true; alive; first = false) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x400);
          break;
        }
        if (units.tickets && rank == 0 && me == 0) ptx::mbar_arrive(units.ask);
        const int ks0 = first_step(unit.slice), ks1 = first_step(unit.slice + 1);
        const int half_n = tl.n >> 1;                       // tokens this CTA loads
        const int row_t = tl.row0 + rank * half_n;
        const int boxes = (half_n + BOX_TOKENS - 1) / BOX_TOKENS;
        const uint32_t t_bytes = GATHER ? half_n * KBYTES : boxes * (BOX_TOKENS * KBYTES);
        const int32_t c0 = GATED ? tl.w_tile * 128 + rank * 64 : tl.w_tile * 256 + rank * 128;
        auto load_weights = [&](int ks, int s) {  // K step ks into stage s; arms the stage for the bytes of all its loads
          const uint32_t sw = ring + s * stage_size, bar0 = bar_full0 + s * 8;
          const int32_t x = ks * (KBYTES / (F8 ? 1 : 2));  // element coordinate along K
          if (rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], 2 * (W_BYTES + t_bytes));
          if constexpr (WMN) {
            ptx::tma_load_3d_pair(sw, &map_w, c0, x, tl.expert, bar0);
            ptx::tma_load_3d_pair(sw + W_BYTES / 2, &map_w, GATED ? c0 + (int32_t)p.n : c0 + 64, x, tl.expert, bar0);
          } else if constexpr (GATED) {
            ptx::tma_load_5d_pair(sw, &map_w, x, 0, 0, c0 >> 4, tl.expert, bar0);
          } else {
            ptx::tma_load_3d_pair(sw, &map_w, x, c0, tl.expert, bar0);
          }
        };
        auto load_tokens = [&](int ks, int s) {
          const uint32_t stok = ring + s * stage_size + W_BYTES, bar0 = bar_full0 + s * 8;
          const int32_t x = ks * (KBYTES / (F8 ? 1 : 2));
          if constexpr (GATHER) {
            auto row = [&](int32_t slot) { return (slot >= 0 && slot < p.numel) ? slot / p.top_k : p.a_rows; };
            for (int r = 0; r < half_n; r += 4) {
              const int4 id = *reinterpret_cast<const int4*>(p.sorted_token_ids + row_t + r);
              ptx::tma_gather4_pair(stok + r * KBYTES, &map_t, x, row(id.x), row(id.y), row(id.z), row(id.w), bar0);
            }
          } else {
            for (int b = 0; b < boxes; ++b)
              ptx::tma_load_2d_pair(stok + b * (BOX_TOKENS * KBYTES), &map_t, x, row_t + b * BOX_TOKENS, bar0);
          }
        };
        int ks = ks0 + mine;
        if (first) {
          // the first tile's weights are on their way before the rows are there: as many K steps as the ring has stages
          const int ahead = early ? min(stages, ks1 - ks0) : 0;
          for (int i = me; i < ahead; i += kProducers) load_weights(ks0 + i, i);
          pdl_wait();
          for (; ks - ks0 < ahead; ks += kProducers) {
            load_tokens(ks, stage);
            advance();
          }
        }
        for (; ks < ks1; ks += kProducers) {
          const long long tp0 = p.profile ? clock64() : 0;
          const bool okp = ptx::mbar_wait(&empty_bar[stage], phase ^ 1);
          if (p.profile) prof_p += clock64() - tp0;
          if (!okp) {
            report(0x100 | stage);
            alive = false;
            break;
          }
          load_weights(ks, stage);
          load_tokens(ks, stage);
          advance();
        }
        mine = ks - ks1;
      }
      if (p.profile && blockIdx.x < 256) g_wait_prof[blockIdx.x * 8 + 3 + 3 * me] = prof_p;
      // drain: what this warp filled has been consumed (in order) before the CTA may end
      if (alive && last_stage >= 0 && !ptx::mbar_wait(&empty_bar[last_stage], last_phase)) report(0x180 | last_stage);
    }
  } else if (warp == kMmaWarp) {
    // ---------------- MMA issuer (CTA 0 only) ----------------
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      bool alive = true;
      long long prof_acc = 0, prof_data = 0;
      const uint32_t ring = ptx::smem_u32(smem);
      const uint64_t db0 = ptx::smem_desc_sw128(ring + W_BYTES);
      // M-major: 64 channels (128 B) x 8 K rows per swizzle atom; the next 8 K rows 1 KB on, the next 64 channels 8 KB on
      const uint64_t da0 = WMN ? ptx::smem_desc_sw128_lbo(ring, W_BYTES / 2, 1024) : ptx::smem_desc_sw128(ring);
      constexpr int a_step = WMN ? (2048 >> 4) : 2;  // one MMA's K: 16 K rows of 128 B, or 32 bytes of each row
      while (alive) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x410);
          break;
        }
        const int ks0 = first_step(unit.slice), ks1 = first_step(unit.slice + 1);
        // bit 15: the M-side operand is M-major
        const uint32_t idesc = ptx::make_idesc(F8 ? /*e4m3*/ 0 : /*bf16*/ 1, 256, (uint32_t)tl.n) | (WMN ? (1u << 15) : 0u);
        const int acc = local & 1;
        const uint32_t acc_phase = (local >> 1) & 1;
        ++local;
        const long long tm0 = p.profile ? clock64() : 0;
        const bool oka = ptx::mbar_wait(&acc_empty[acc], acc_phase ^ 1);
        if (p.profile) prof_acc += clock64() - tm0;
        if (!oka) {
          report(0x200 | acc);
          alive = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
        for (int ks = ks0; ks < ks1; ++ks) {
          const long long tm1 = p.profile ? clock64() : 0;
          const bool okd = ptx::mbar_wait(&full_bar[stage], phase);
          if (p.profile) prof_data += clock64() - tm1;
          if (!okd) {
            report(0x240 | stage);
            alive = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint64_t da = da0 + (uint64_t)(stage * (stage_size >> 4)), db = db0 + (uint64_t)(stage * (stage_size >> 4));
#pragma unroll
          for (int kk = 0; kk < KBYTES / 32; ++kk) {
            if constexpr (F8) ptx::mma_f8f6f4_ss_pair(d_tmem, da + a_step * kk, db + 2 * kk, idesc, ((ks - ks0) | kk) != 0);
            else ptx::mma_f16_ss_pair(d_tmem, da + a_step * kk, db + 2 * kk, idesc, ((ks - ks0) | kk) != 0);
          }
          ptx::mma_commit_both(&empty_bar[stage]);  // the stage is free in both CTAs once these MMAs have read it
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (alive) ptx::mma_commit_both(&acc_full[acc]);
      }
      if (p.profile && blockIdx.x < 256) {
        g_wait_prof[blockIdx.x * 8 + 0] = local;
        g_wait_prof[blockIdx.x * 8 + 1] = prof_acc;
        g_wait_prof[blockIdx.x * 8 + 2] = prof_data;
      }
    }
  } else if (warp == kMmaWarp + 1) {
    // ---------------- the worker's units ----------------
    UnitPlan plan;
    plan.init((int64_t)table[3 * p.num_experts] * p.w_tiles, k_steps, p.split_max, workers, worker);
    auto unit_at = [&](int64_t it, int4* d) {
      int64_t tile;
      int ks0, ks1;
      PairUnit u;
      const bool any = plan.get(it, &tile, &ks0, &ks1, &u.slice);
      *d = make_int4(0, 0, 0, 0);
      if (any) {
        u.tl = pair_locate(tile, p.w_tiles, p.group, p.num_experts, table);
        u.log2_s = plan.is_split(it) ? 31 - __clz(plan.S) : 0;
        u.b = plan.b;
        *d = u.pack();
      }
      return any;
    };
    int4* list = const_cast<int4*>(units.units);
    int4 d;
    if (!units.tickets) {
      bool more = true;
      for (int half = 0; more; ++half) {
        if (!units.wait_half(half)) {
          report(0x430);
          break;
        }
        more = __all_sync(0xffffffffu, unit_at((int64_t)half * kListUnits + lane, &d));
        list[(half & 1) * kListUnits + lane] = d;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&units.full[(half & 1) * kListUnits]);
      }
    } else if (rank == 0) {
      bool more = true;
      for (int i = 0, ticket = worker; more; ++i) {
        if (i) {
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_relaxed(units.ask, (i - 1) & 1))) {
            report(0x431);
            break;
          }
          if (lane == 0) ticket = workers + atomicAdd(p.tickets, 1);
          ticket = __shfl_sync(0xffffffffu, ticket, 0);
        }
        if (i % kListUnits == 0 && !units.wait_half(i / kListUnits)) {
          report(0x432);
          break;
        }
        plan.b = ticket % workers;
        more = unit_at(ticket / workers, &d);
        const int slot = i % (2 * kListUnits);
        if (lane < 2) ptx::st_async_16(ptx::mapa(ptx::smem_u32(list + slot), lane), d, ptx::mapa(ptx::smem_u32(&units.full[slot]), lane));
      }
    }
  } else {
    // ---------------- epilogue (both CTAs, each its CTA's 128 weight rows) ----------------
    pdl_entry_late();
    const int quarter = warp & 3, half = warp >> 2;
    const int g = lane >> 2, t = lane & 3;
    uint8_t* strip = strips + warp * STRIP_BYTES;
    int local = 0;
    bool alive = true;
    long long prof_wait = 0, prof_busy = 0;
    while (alive) {
      const bool waits = units.waits();
      int got = units.next<true>(&unit);
      if (waits && any_of_four_warps(1 + half, got < 0)) got = -1;  // warps that meet at a barrier below leave together
      if (got <= 0) {
        if (got < 0) report(0x420);
        break;
      }
      const int slice = unit.slice, S = 1 << unit.log2_s;
      const int acc = local & 1;
      const uint32_t acc_phase = (local >> 1) & 1;
      ++local;
      const int chunks = tl.n >> 4;  // 16-token chunks; this warp takes those that are `half` modulo HALVES
      // token f = 16 * c + u of the warp's c-th chunk sits in register f / 32 of lane f % 32
      constexpr int REGS = 8 / HALVES;
      int32_t slot_r[REGS];
      float rs_r[REGS];
#pragma unroll
      for (int r = 0; r < REGS; ++r) {
        const int f = r * 32 + lane;
        const int tok = (HALVES * (f >> 4) + half) * 16 + (f & 15);
        slot_r[r] = -1;
        rs_r[r] = 1.0f;
        if (tok < tl.cols) {
          const int32_t s = p.sorted_token_ids[tl.row0 + tok];
          if (s >= 0 && s < p.numel) {
            slot_r[r] = s;
            if (p.row_scale) rs_r[r] = p.row_scale[s];
            if constexpr (F8) rs_r[r] *= p.a_scale_gather ? p.a_scale[s / p.top_k] : p.a_scale[tl.row0 + tok];
          }
        }
      }
      // first output channel of this warp, and per-channel factors / biases of its rows: gated {gate g, gate g+8, up g,
      // up g+8}, plain {g, g+8, g+16, g+24}
      const int quarter_ch = WMN ? 32 * (quarter & 1) + 16 * (quarter >> 1) : 16 * quarter;
      const int ch0 = GATED ? tl.w_tile * 128 + rank * 64 + quarter_ch : tl.w_tile * 256 + rank * 128 + quarter * 32;
      float cv[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr ((F8 || EXTRA) && !WMN) {
        const float* vec = F8 ? p.w_scale : p.bias;
        if (vec) {
          vec += (int64_t)tl.expert * p.w_rows;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int64_t c = GATED ? ch0 + g + 8 * (i & 1) : ch0 + g + 8 * i;
            if (c < p.n) cv[i] = GATED ? vec[c * p.vec_step + (i >= 2 ? p.vec_up : 0)] : vec[c];
          }
        }
      }
      const long long te0 = p.profile ? clock64() : 0;
      const bool split = S > 1;
      bool oke = warp_wait_relaxed(&acc_full[acc], acc_phase);
      // warps that meet at a barrier below leave together or not at all
      if (split || (GATED && WMN)) oke = !any_of_four_warps(1 + half, !oke);
      const long long te1 = p.profile ? clock64() : 0;
      prof_wait += te1 - te0;
      if (!oke) {
        report(0x300 | acc);
        alive = false;
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      // fragment (slice o, chunk j) of this thread: four float4, 512 bytes apart so that a warp stores whole lines
      auto partial = [&](int o, int j) {
        return reinterpret_cast<float4*>(p.split_partials) +
               ((((int64_t)(unit.b - slice + o) * 2 + rank) * 16 + j) * 4 + quarter) * 128 + lane;
      };
      bool finish = true;  // these four warps run the epilogue of their chunks
      if (split) {
#pragma unroll 1
        for (int j = half; j < chunks; j += HALVES) {
          uint32_t lo[8], hi[8];
          ptx::tmem_ld_16x256b_x2(taddr + j * 16, lo);
          ptx::tmem_ld_16x256b_x2(taddr + (16u << 16) + j * 16, hi);
          ptx::tmem_ld_wait();
          float4* dst = partial(slice, j);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t* v = q < 2 ? lo + 4 * q : hi + 4 * (q - 2);
            __stcg(dst + 32 * q, make_float4(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]),
                                             __uint_as_float(v[3])));
          }
        }
        __threadfence();  // the partials are visible device-wide before these warps count as arrived
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        finish = any_of_four_warps(1 + half, quarter == 0 && lane == 0 &&
                                                 atomicAdd(p.split_counters + ((unit.b >> unit.log2_s) * 2 + rank) * 4 + half, 1) == S - 1);
        __threadfence();  // the other slices' partials are read after the count
      }
      // the next chunk's TMEM read-out is in flight while a chunk is stored
      const int c_end = finish ? chunks : 0;
      int j = half;
      uint32_t nlo[8], nhi[8];
      if (j < c_end && !split) {
        ptx::tmem_ld_16x256b_x2(taddr + j * 16, nlo);                // rows 0-15 of the quarter (gated: gate)
        ptx::tmem_ld_16x256b_x2(taddr + (16u << 16) + j * 16, nhi);  // rows 16-31 (gated: up)
      }
#pragma unroll 1
      for (; j < c_end; j += HALVES) {
        uint32_t lo[8], hi[8];
        if (split) {  // all slices' partials in slice order, whoever adds them
#pragma unroll
          for (int i = 0; i < 8; ++i) lo[i] = hi[i] = 0u;
#pragma unroll 1
          for (int o = 0; o < S; ++o) {
            const float4* src = partial(o, j);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 v = __ldcg(src + 32 * q);
              uint32_t* d = q < 2 ? lo + 4 * q : hi + 4 * (q - 2);
              d[0] = __float_as_uint(__uint_as_float(d[0]) + v.x);
              d[1] = __float_as_uint(__uint_as_float(d[1]) + v.y);
              d[2] = __float_as_uint(__uint_as_float(d[2]) + v.z);
              d[3] = __float_as_uint(__uint_as_float(d[3]) + v.w);
            }
          }
        } else {
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            lo[i] = nlo[i];
            hi[i] = nhi[i];
          }
          if (j + HALVES < c_end) {
            ptx::tmem_ld_16x256b_x2(taddr + (j + HALVES) * 16, nlo);
            ptx::tmem_ld_16x256b_x2(taddr + (16u << 16) + (j + HALVES) * 16, nhi);
          }
        }
        // the chunk's 16 slots and row scales, from the lanes that hold them
        const int c = j / HALVES;
        int32_t slot_c = slot_r[0];
        float rs_c = rs_r[0];
#pragma unroll
        for (int r = 1; r < REGS; ++r) {
          if ((c >> 1) == r) {
            slot_c = slot_r[r];
            rs_c = rs_r[r];
          }
        }
        const int src_lane = (c & 1) * 16;
        float rs[4];  // columns 2t, 2t+1, 8+2t, 9+2t
#pragma unroll
        for (int q = 0; q < 4; ++q) rs[q] = __shfl_sync(0xffffffffu, rs_c, src_lane + (q >> 1) * 8 + 2 * t + (q & 1));
        if constexpr (GATED) {
          if constexpr (WMN) {
            // M-major gate rows are in lanes 0-63 and the up rows of the same channels in lanes 64-127: two warps swap halves
            // through shared memory, lane by lane.  The gate warp finishes its first 16 channels, the up warp the other 16.
            // (Four warps that met twice a chunk and read back by token, eight such warps: 8500 cycles for 128 tokens, more than
            // the 20 K steps of the reference shape.  1024 tokens of it through the operator: 348 -> 326 us.)
            const bool gate = quarter < 2;
            float4* mine = reinterpret_cast<float4*>(strip) + lane;
            const float4* theirs = reinterpret_cast<const float4*>(strips + (warp ^ 2) * STRIP_BYTES) + lane;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint32_t o[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) o[i] = gate ? hi[4 * q + i] : lo[4 * q + i];
              mine[32 * q] = make_float4(__uint_as_float(o[0]), __uint_as_float(o[1]), __uint_as_float(o[2]), __uint_as_float(o[3]));
            }
            pair_of_warps_sync(half * 2 + (quarter & 1));
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const float4 v = theirs[32 * q];
              const uint32_t got[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (gate) hi[4 * q + i] = got[i];
                else lo[4 * q + i] = got[i];
              }
            }
            pair_of_warps_sync(half * 2 + (quarter & 1));  // both have read: the strips are free
          }
          uint32_t m[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {  // q = 2 * (column group) + (row half)
            const int i = 4 * (q >> 1) + 2 * (q & 1);
            float o[2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              const float gv = __uint_as_float(lo[i + v]), uv = __uint_as_float(hi[i + v]), r = rs[2 * (q >> 1) + v];
              if constexpr (EXTRA)
                o[v] = gated_output<true>(gv, uv, cv[q & 1], cv[2 + (q & 1)], r, p.activation, p.act_alpha, p.act_limit);
              else if constexpr (F8)  // (accumulator * row scale) * channel scale, then the activation
                o[v] = act_mul_fast(gv * r * cv[q & 1], uv * r * cv[2 + (q & 1)], p.activation);
              else
                o[v] = act_mul_fast(gv * r, uv * r, p.activation);
            }
            m[q] = pack_bf16x2(o[0], o[1]);
          }
          strip_put16(strip, 48, 0, lane, m);
          strip_store_sorted(strip, lane, reinterpret_cast<__nv_bfloat16*>(p.out) + (int64_t)(tl.row0 + j * 16) * p.n, p.n, ch0,
                             tl.cols - j * 16);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = 4 * (q >> 1) + 2 * (q & 1);
              const uint32_t* a = h ? hi : lo;
              const float v0 = __uint_as_float(a[i]), v1 = __uint_as_float(a[i + 1]);
              const float r0 = rs[2 * (q >> 1)], r1 = rs[2 * (q >> 1) + 1], c0 = cv[2 * h + (q & 1)];
              if constexpr (F8) m[q] = pack_bf16x2(v0 * r0 * c0, v1 * r1 * c0);
              else m[q] = pack_bf16x2((v0 + c0) * r0, (v1 + c0) * r1);
            }
            strip_put16(strip, 80, 16 * h, lane, m);
          }
          strip_store_slots(strip, lane, p.out, p.out_rows, p.n, ch0, __shfl_sync(0xffffffffu, slot_c, src_lane + (lane >> 2)),
                            __shfl_sync(0xffffffffu, slot_c, src_lane + 8 + (lane >> 2)));
        }
      }
      // the accumulator may be overwritten from here on: tell CTA 0's MMA warp
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(ptx::smem_u32(&acc_empty[acc]) & ~ptx::kPeerRankBit);
      if constexpr (GATED) {
        if (p.zero_padding && tl.last && slice == 0)
          zero_block_rows(tl, p.out, p.n, tl.w_tile * 128 + rank * 64, 2, threadIdx.x, kEpiWarps * 32);
      }
      if (p.profile) prof_busy += clock64() - te1;
    }
    if (p.out_rows) __threadfence_system();  // rows stored to a peer are complete before the kernel ends
    if (p.profile && threadIdx.x == 0 && blockIdx.x < 256) {
      g_wait_prof[blockIdx.x * 8 + 4] = prof_wait;
      g_wait_prof[blockIdx.x * 8 + 5] = prof_busy;
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();  // nobody signals into a CTA that has left, and both are done with TMEM
  if (warp == kMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// ---- host side ----------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

}  // namespace

int encode_tensor_map(CUtensorMap* map, const void* base, int elem_bytes, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
           const cuuint32_t* box, bool weights, const char* what) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(FMOE_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, (cuuint32_t)rank,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B,
                  weights ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FMOE_ERR_CUDA, "cuTensorMapEncodeTiled (%s) failed with code %d", what, (int)r);
  return FMOE_OK;
}

// SM count of the current device (cached per device ordinal).
int device_sm_count() {
  static std::mutex mu;
  static int sm_count[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev < 0 || dev >= kMaxDevices) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (sm_count[dev] == 0) cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
  return sm_count[dev];
}

// Host-side view of the work-unit plan (the same code the kernels run), for tests.
int tail_plan_unit(int64_t total_tiles, int k_steps, int max_split, int grid, int cta, int64_t it, int64_t* out) {
  UnitPlan plan;
  plan.init(total_tiles, k_steps, max_split, grid, cta);
  int64_t tile = 0;
  int ks0 = 0, ks1 = 0, slice = 0;
  if (!plan.get(it, &tile, &ks0, &ks1, &slice)) return 0;
  out[0] = tile;
  out[1] = ks0;
  out[2] = ks1;
  out[3] = slice;
  out[4] = plan.is_split(it) ? plan.S : 1;
  return 1;
}

int64_t gemm_pair_split_workspace_bytes() {
  const int sms = device_sm_count();
  return kSplitCounters * 4 + (int64_t)std::min(std::max(sms, 1), 256) * 128 * 256 * 4;
}

// tokens: row-major [rows, cols]; box = 128 bytes x box_rows
int pair_map_tokens(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int elem_bytes, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * elem_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(KBYTES / elem_bytes), (cuuint32_t)box_rows};
  return encode_tensor_map(map, base, elem_bytes, 2, dims, strides, box, false, "tokens");
}

// weights [E, rows, K], K contiguous.  gated: rows = n gate rows then n up rows; the box takes 4 groups of 16 gate rows and
// the 16 matching up rows (K, 16 rows, gate/up, row groups, expert: rows past n read as zeros); interleaved: gate and up rows
// alternate, the box is the same.  plain: rows = n, 128 rows.
int pair_map_weights(CUtensorMap* map, const void* base, int64_t experts, int64_t n, int64_t k, int elem_bytes, bool gated,
                     bool interleaved) {
  const cuuint64_t row = (cuuint64_t)k * elem_bytes;
  if (gated) {
    const cuuint64_t dims[5] = {(cuuint64_t)k, 16, 2, (cuuint64_t)(n / 16), (cuuint64_t)experts};
    const cuuint64_t strides[4] = {interleaved ? row * 2 : row, interleaved ? row : row * n, interleaved ? row * 32 : row * 16,
                                   row * 2 * n};
    const cuuint32_t box[5] = {(cuuint32_t)(KBYTES / elem_bytes), 16, 2, 4, 1};
    return encode_tensor_map(map, base, elem_bytes, 5, dims, strides, box, true, "gate/up weights");
  }
  const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)n, (cuuint64_t)experts};
  const cuuint64_t strides[2] = {row, row * n};
  const cuuint32_t box[3] = {(cuuint32_t)(KBYTES / elem_bytes), 128, 1};
  return encode_tensor_map(map, base, elem_bytes, 3, dims, strides, box, true, "down weights");
}

// bf16 weights [E, K, w_rows] with w_rows contiguous; box = 64 channels (128 bytes, the swizzle width) x 64 K rows.
int pair_map_weights_nmajor(CUtensorMap* map, const void* base, int64_t experts, int64_t k, int64_t w_rows) {
  const cuuint64_t dims[3] = {(cuuint64_t)w_rows, (cuuint64_t)k, (cuuint64_t)experts};
  const cuuint64_t strides[2] = {(cuuint64_t)w_rows * 2, (cuuint64_t)w_rows * (cuuint64_t)k * 2};
  const cuuint32_t box[3] = {64, 64, 1};
  return encode_tensor_map(map, base, 2, 3, dims, strides, box, true, "N-major weights");
}

namespace {

template <bool GATED, bool F8, bool EXTRA, bool WMN, bool GATHER>
int launch(const GemmParams& g, cudaStream_t st) {
  constexpr int ELEM = F8 ? 1 : 2;
  constexpr int MAX_SMEM = smem_bytes(1024);
  auto kernel = grouped_gemm_pair_kernel<GATED, F8, EXTRA, WMN, GATHER>;
  const int smem = smem_bytes(g.num_experts);
  static PerDeviceOnce once_attr;  // the opt-in to > 48 KB of dynamic shared memory is per device
  const cudaError_t attr_err = per_device_once(once_attr, [&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
  });
  if (attr_err != cudaSuccess)
    return fail(FMOE_ERR_CUDA, "cudaFuncSetAttribute(smem=%d) failed: %s", MAX_SMEM, cudaGetErrorString(attr_err));

  const int64_t w_rows = GATED ? 2 * g.n : g.n;
  const bool interleaved = GATED && g.w_layout == FMOE_W_INTERLEAVED;
  CUtensorMap map_t, map_w;
  int rc = pair_map_tokens(&map_t, g.a, g.a_rows, g.k, ELEM, GATHER ? 1 : BOX_TOKENS);
  if (rc) return rc;
  if constexpr (WMN) rc = pair_map_weights_nmajor(&map_w, g.w, g.num_experts, g.k, w_rows);
  else rc = pair_map_weights(&map_w, g.w, g.num_experts, g.n, g.k, ELEM, GATED, interleaved);
  if (rc) return rc;

  PairParams p;
  p.sorted_token_ids = g.sorted_token_ids;
  p.expert_ids = g.expert_ids;
  p.num_tokens_post_padded = g.num_tokens_post_padded;
  p.expert_table = g.expert_table;
  p.early = g.expert_table && g.behind_late_trigger;
  p.row_scale = g.row_scale;
  p.a_scale = g.a_scale;
  p.a_scale_gather = g.a_scale_gather;
  p.w_scale = g.w_scale;
  p.bias = g.bias;
  p.vec_step = interleaved ? 2 : 1;
  p.vec_up = interleaved ? 1 : (int32_t)g.n;
  p.act_alpha = g.act_alpha;
  p.act_limit = g.act_limit;
  p.out = g.out;
  p.out_rows = GATED ? nullptr : g.out_rows;
  p.numel = g.numel;
  p.n = g.n;
  p.w_rows = w_rows;
  p.num_experts = g.num_experts;
  p.k_steps = (int)ceil_div<int64_t>(g.k * ELEM, KBYTES);
  p.w_tiles = (int)ceil_div<int64_t>(g.n, GATED ? 128 : 256);
  p.max_blocks = (int)g.max_blocks;
  p.activation = g.activation;
  p.top_k = g.top_k;
  p.a_rows = (int32_t)g.a_rows;
  p.zero_padding = !g.skip_padding;
  p.token_tile = g.token_tile ? g.token_tile : pick_token_tile(g.numel, g.num_experts, g.dtype == FMOE_E4M3);
  p.stage_bytes = stage_bytes(p.token_tile);
  p.stages = std::min(RING_BYTES / p.stage_bytes, MAX_STAGES);
  p.group = pick_group_m(p.token_tile, g.k * ELEM);
  static const bool profile = getenv("FMOE_TC_PROFILE") != nullptr;
  p.profile = profile;

  const int64_t max_tiles = g.max_blocks * ceil_div(128, p.token_tile) * p.w_tiles;
  const int sms = device_sm_count();
  const int workers = (int)std::max<int64_t>(1, std::min<int64_t>((sms > 0 ? sms : 148) / 2, max_tiles));
  p.split_partials = nullptr;
  p.split_counters = nullptr;
  p.split_max = 0;
  p.tickets = nullptr;
  const char* split_env = getenv("FMOE_TC_SPLIT_TAIL");  // "0": off (read per launch, tests flip it)
  const bool split_off = split_env && split_env[0] == '0';
  const bool split_fits = g.split_ws_bytes >= kSplitCounters * 4 + (int64_t)workers * 2 * 128 * 256 * 4 && workers <= 128;
  if (g.split_ws && !split_off && split_fits && aligned16(g.split_ws)) {
    p.split_partials = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(g.split_ws) + kSplitCounters * 4);
    p.split_max = GATED ? 4 : 8;
    if (g.split_counters) {
      p.split_counters = g.split_counters;
    } else {
      p.split_counters = reinterpret_cast<int32_t*>(g.split_ws);
      FMOE_CUDA_OK(cudaMemsetAsync(g.split_ws, 0, kSplitCounters * 4, st));
    }
  }
  // Units by ticket from 800 K steps a worker on (by the rows an expert has on average), and where there is a zeroed word.  Layers
  // dealt / by ticket in us: Mixtral 2048 tokens 1407 / 1390, 3000 2054 / 1919, 3500 2419 / 2196, 4096 2650 / 2516, 8192 5146 /
  // 4804; Qwen3 16384 tokens 1478 / 1425; DeepSeek-V3 per channel 8192 tokens 4251 / 4047, 2048 1855 / 1851, 16 544 / 540.  Below,
  // what a ticket takes shows and there is no drift to save: half of Mixtral 333 tokens 266.6 / 268.2, Mixtral 19 tokens 437.2 /
  // 439.7, a quarter of Qwen3 (down GEMM of 3 K steps a tile) 387 / 397.
  int32_t* counters = g.split_counters ? g.split_counters : p.split_counters;
  const int64_t active = std::min<int64_t>(g.num_experts, g.numel);
  const int64_t tiles = std::max(active, g.numel / p.token_tile + active / 2) * p.w_tiles;
  if (counters && workers <= kMaxTicketWorkers && tiles * p.k_steps >= 800 * workers) p.tickets = counters + kSplitCounters - 1;
  launch_pdl(kernel, dim3(2 * workers), dim3(kThreads), smem, st, map_t, map_w, p);
  return launch_status("grouped_gemm_pair_kernel");
}

}  // namespace

bool gemm_pair_supports(const GemmParams& p, bool gated) {
  const bool f8 = p.dtype == FMOE_E4M3 && p.scale_mode == FMOE_SCALE_CHANNEL;
  if ((p.dtype != FMOE_BF16 && !f8) || p.out_dtype != FMOE_BF16) return false;
  // e4m3 with per-row / per-channel scales: plain kernels, K-major weights, sorted input rows
  if (f8 && (p.a_gather || p.bias || p.w_layout != FMOE_W_K_MAJOR || !p.a_scale || !p.w_scale || !aligned16(p.w_scale) ||
             (gated && p.activation == FMOE_ACT_SWIGLU_OAI)))
    return false;
  if (p.block_size != 128) return false;
  // gather mode: gate/up GEMM only; one int4 of sorted ids per lane
  if (p.a_gather && (!gated || p.top_k < 1 || !aligned16(p.sorted_token_ids))) return false;
  if (p.w_layout != FMOE_W_K_MAJOR && p.w_layout != FMOE_W_N_MAJOR && !(p.w_layout == FMOE_W_INTERLEAVED && gated)) return false;
  // weights in the reference operator's [E, K, N] layout: plain kernels only (no row gather, bias or swiglu_oai)
  if (p.w_layout == FMOE_W_N_MAJOR && (p.a_gather || p.bias || (gated && p.activation == FMOE_ACT_SWIGLU_OAI))) return false;
  if (p.k <= 0 || (p.k * (f8 ? 1 : 2)) % 16 != 0) return false;  // TMA row stride must be a multiple of 16 bytes
  if (p.n <= 0 || p.n % 32 != 0) return false;  // gate/up row groups of 16, 16-byte stores
  if (!aligned16(p.a) || !aligned16(p.w) || !(aligned16(p.out) && (p.out || (!gated && p.out_rows)))) return false;
  if ((int64_t)p.num_experts * (gated ? 2 * p.n : p.n) >= (1ll << 31) || p.a_rows >= (1ll << 31)) return false;
  if (p.max_blocks >= (1ll << 24) || p.num_experts > 1024) return false;
  return true;
}

int gemm_pair(const GemmParams& p, bool gated, cudaStream_t st) {
  if (!gemm_pair_supports(p, gated))
    return fail(FMOE_ERR_UNSUPPORTED,
                "tcgen05 gemm: needs bf16 in/out (or e4m3 in with per-channel scales), block_size 128, input-row gather only for the gate/up gemm, "
                "n %% %d == 0, 16-byte aligned pointers (got dtype=%d block=%d a_gather=%d n=%lld k=%lld)",
                32, p.dtype, p.block_size, p.a_gather, (long long)p.n, (long long)p.k);
  if (p.max_blocks <= 0) return FMOE_OK;
  const bool extra = p.bias != nullptr || (gated && p.activation == FMOE_ACT_SWIGLU_OAI);
  //                                      GATED  F8    EXTRA  WMN    GATHER
  if (p.dtype == FMOE_E4M3)
    return gated ? launch<true, true, false, false, false>(p, st) : launch<false, true, false, false, false>(p, st);
  if (p.w_layout == FMOE_W_N_MAJOR)
    return gated ? launch<true, false, false, true, false>(p, st) : launch<false, false, false, true, false>(p, st);
  if (p.a_gather) return extra ? launch<true, false, true, false, true>(p, st) : launch<true, false, false, false, true>(p, st);
  if (gated) return extra ? launch<true, false, true, false, false>(p, st) : launch<true, false, false, false, false>(p, st);
  return extra ? launch<false, false, true, false, false>(p, st) : launch<false, false, false, false, false>(p, st);
}

namespace {
// Self-test of the time-out path: waits on a barrier that nobody signals, with a short limit.
__global__ void bounded_wait_selftest_kernel(long long limit_cycles) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bar, 1);
    ptx::fence_barrier_init();
  }
  __syncthreads();
  if (!ptx::mbar_wait_limit(&bar, 0, limit_cycles) && threadIdx.x == 0) report(0xE00);
}
}  // namespace

int launch_bounded_wait_selftest(long long limit_cycles, cudaStream_t st) {
  bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(limit_cycles);
  return launch_status("bounded_wait_selftest_kernel");
}

int read_wait_profile(long long* host_out, int n) {
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(host_out, g_wait_prof, sizeof(long long) * (size_t)n));
  return FMOE_OK;
}

int status_word_fp8(int* out, bool clear);
int status_word_ep(int* out, bool clear);
int status_word_decode(int* out, bool clear);
int status_word_align(int* out, bool clear);

// First non-zero status word of the translation units that keep one (tcgen05 kernels, decode layer,
// expert-parallel exchange, routing triple); all are cleared.
int read_and_clear_device_status(cudaStream_t st, int* status_out) {
  int zero = 0, a = 0, b = 0, c = 0, d = 0, e = 0;
  FMOE_CUDA_OK(cudaStreamSynchronize(st));
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(&a, g_device_status, sizeof(int)));
  if (a != 0) FMOE_CUDA_OK(cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int)));
  int rc = status_word_fp8(&b, true);
  if (rc) return rc;
  rc = status_word_decode(&c, true);
  if (rc) return rc;
  rc = status_word_ep(&d, true);
  if (rc) return rc;
  rc = status_word_align(&e, true);
  if (rc) return rc;
  *status_out = a ? a : (b ? b : (c ? c : (d ? d : e)));
  return FMOE_OK;
}

}  // namespace fmoe
