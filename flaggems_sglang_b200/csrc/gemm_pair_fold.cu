// Grouped GEMM on CTA pairs for e4m3 operands with 128x128 weight scales and 1x128 activation scales.
//
// tcgen05 accumulates in fp32 inside TMEM and cannot apply a different scale to every 128-wide K block, so every K block
// (128 bytes = 128 e4m3 = one scale block) is multiplied into a FRESH TMEM partial (4 MMAs of K = 32, the first one
// overwriting), and the fold warps add it into register accumulators:
//     acc[channel, token] += partial[channel, token] * (a_scale[token, kb] * w_scale[channel / 128, kb])
//
// Two kernels: the narrow one (64-token tiles, few rows per expert) and the wide one (below).  The narrow one:
//   tile      : 256 weight rows (128 per CTA) x up to 64 tokens of one expert, as in gemm_pair.cu (same tile order, same
//               row interleave of gate and up, same transposed stores)
//   TMEM      : 512 columns per CTA as eight partials of 64 tokens: the MMAs of the next K blocks run while one is folded
//   warps 0-15: fold + epilogue.  Warps 0-7 fold the K blocks of even step, 8-15 those of odd step, so that one block's TMEM
//               reads and waits run beside the other's FMAs; the two sums meet in the epilogue.  Warp w reads TMEM lanes
//               32 * (w % 4).. and the 16-token pieces w / 4 % 2 and 2 further.  The 16 x 256b read-out puts two tokens of
//               one channel side by side, which is what the packed fma.rn.f32x2 takes with one pair of factors for two
//               channels.  A partial is handed back when it is in registers, before the FMAs.  (All sixteen warps on every
//               block: 722 SM cycles per K block; this split 572.  DeepSeek-V3, 128 tokens 1361 -> 1245 us, 1024 tokens
//               2190 -> 2005 us per layer.)  The gate/up output is fp32, for the quantiser behind it
//   warp 16   : TMA producer      warp 17 : MMA issuer (CTA 0)
//   warps 18-19: factors (and warp 18 the list of the worker's tiles).  For four K blocks at a time they multiply the tokens'
//               scales with the tile's one or two weight scales and leave the products in a 4-slot ring in shared memory, next
//               to the tile's slots and row weights: the fold warps read one 8-byte pair per two tokens and keep no pointers
// What bounds it: HBM (the weights stream through a ring of 20 KB stages) up to about 8 rows per expert, the fold above.
#include "pair.cuh"
#include "rows.cuh"

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace fmoe {

// This translation unit's status word (device code is not linked across files); read by status_word_fp8().
__device__ int g_device_status_fp8 = 0;
// Wait-time profile of the instrumented build of the kernel (FMOE_TC_PROFILE=1): per CTA
// {tiles, fold waits for the MMAs, fold busy, fold waits for staged scales, epilogue, kernel cycles, MMA warp waits for a
// partial, MMA warp waits for data};
// [0]: down GEMM, [1]: gate/up GEMM
__device__ long long g_wait_prof_fp8[2 * 256 * 8];

namespace {

constexpr int KBYTES = 128;
constexpr int W_BYTES = 128 * KBYTES;
constexpr int TMEM_COLS = 512;
constexpr int kFoldWarps = 16;
constexpr int kThreads = (kFoldWarps + 4) * 32;
constexpr int kFoldRegs = 104, kOtherRegs = 64;  // per thread, out of the launch's 20 * 96 per lane (setmaxnreg)
constexpr int BOX_TOKENS = 32;
constexpr int SC_SLOTS = 4;                      // factor ring: slots of 4 K blocks
constexpr int META_TILES = 8;                    // more than the SC_SLOTS tiles that the factor warps may be ahead of the fold
constexpr int BAR_BYTES = 512;
constexpr int kMaxSmem = 227 * 1024;
// Geometry of the narrow kernel
constexpr int TOK = 64;
template <bool GATED>
struct Geo {
  static constexpr int STAGE_BYTES = W_BYTES + TOK / 2 * KBYTES;
  static constexpr int STAGES = GATED ? 8 : 7;
  static constexpr int BUFS = TMEM_COLS / TOK;                 // TMEM partials
  static constexpr int KB_BYTES = (GATED ? 2 : 1) * TOK * 4;   // factors of one K block
  static constexpr int STRIP_BYTES = GATED ? 16 * 48 : 16 * 80;
  static constexpr int FACTOR_BYTES = SC_SLOTS * 4 * KB_BYTES;
  static constexpr int EX_BYTES = 2 * 1024;                    // per fold warp: sums on their way to the partner warp
  static constexpr int META_BYTES = GATED ? 0 : META_TILES * TOK * 8;  // slots and row weights of the tile's tokens
  static constexpr int bytes(int num_experts) {
    return STAGES * STAGE_BYTES + BAR_BYTES + kListBytes + kFoldWarps * (STRIP_BYTES + EX_BYTES) + FACTOR_BYTES + META_BYTES +
           pair_table_bytes(num_experts);
  }
};
static_assert(Geo<true>::bytes(1024) <= kMaxSmem && Geo<false>::bytes(1024) <= kMaxSmem, "shared memory");

struct FoldParams {
  const int32_t* sorted_token_ids;
  const int32_t* expert_ids;
  const int32_t* num_tokens_post_padded;
  const int32_t* expert_table;
  const float* row_scale;
  const float* a_scale;  // [a_rows, kblocks], or [tokens, kblocks] (a_scale_gather)
  const float* w_scale;  // [E, w_rows/128, kblocks]
  void* out;
  void* const* out_rows;  // down projection: optional per-slot row addresses (may be peer memory)
  int64_t numel;
  int64_t n;
  int64_t w_rows;
  int32_t a_scale_gather;
  int32_t top_k;
  int32_t num_experts;
  int32_t kblocks;
  int32_t w_tiles;
  int32_t max_blocks;
  int32_t activation;
  int32_t group;
  int32_t zero_padding;
  int32_t out_dtype;  // gate/up: FMOE_F32, FMOE_BF16 or (wide) FMOE_E4M3 with out_scale
  float* out_scale;   // [rows, n / 128]
  int32_t min_rows, max_rows;  // experts of this launch
  bool stores_of_32;           // rows of the output start at multiples of 32 bytes
  bool early;                  // the table is complete when the kernel starts
  bool by_expert;              // narrow, fp32 gate/up output: kNarrowRows rows per expert instead of one per position
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_device_status_fp8, 0, code); }
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity));
}

// acc (two packed floats) += v * f, both lanes
__device__ __forceinline__ void fma2(unsigned long long& acc, uint32_t v0, uint32_t v1, unsigned long long ff) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(v0), "r"(v1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(v), "l"(ff));
}
__device__ __forceinline__ float lds32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// weight of the tile's token u when top-k weights go to the gate/up GEMM
__device__ __forceinline__ float row_weight(const FoldParams& p, const PairTile& tl, int u) {
  const int32_t s = u < tl.cols ? p.sorted_token_ids[tl.row0 + u] : -1;
  return (s >= 0 && s < p.numel) ? p.row_scale[s] : 1.0f;
}
__device__ __forceinline__ unsigned long long lds64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}

// One 32-byte store where the destination is aligned to it, else two of 16 bytes.  The wide kernel's lanes store to 32 rows at
// once, so that every instruction touches 32 lines whatever it writes.  (Down GEMM, 64 experts of 512 rows,
// H = 7168, I = 2048: 650 us with 16-byte stores, 550 with 32.)
__device__ __forceinline__ void store_32_bytes(void* dst, const uint32_t (&w)[8], bool whole) {
  if (whole) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
                 "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}
// 16 values times s as bf16
__device__ __forceinline__ void store16(__nv_bfloat16* dst, const float* v, float s, bool whole) {
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = pack_bf16x2(v[2 * j] * s, v[2 * j + 1] * s);
  store_32_bytes(dst, w, whole);
}

__device__ __forceinline__ void sts64(uint32_t addr, unsigned long long v) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

// PROF: instrumented build with wait-time counters (reading the clock is slow enough to distort the fold loop).
// MOVE: registers move from the other warps to the fold warps (setmaxnreg); see launch().
template <bool GATED, bool PROF, bool MOVE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
grouped_gemm_pair_fold_kernel(const __grid_constant__ CUtensorMap map_t, const __grid_constant__ CUtensorMap map_w,
                              const FoldParams p) {
  using G = Geo<GATED>;
  constexpr int PIECES = TOK / 32;  // 16-token pieces per fold warp: half and half + 2
  constexpr int STAGES = G::STAGES, STAGE_BYTES = G::STAGE_BYTES, BUFS = G::BUFS, KB_BYTES = G::KB_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];  // aligned by declaration: every address below is a constant
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full_bar = bars;                            // [STAGES] used in CTA 0: both CTAs' loads -> MMA
  uint64_t* empty_bar = bars + STAGES;              // [STAGES] per CTA: MMA -> producer
  uint64_t* part_full = bars + 2 * STAGES;          // [bufs] per CTA: MMA -> fold
  uint64_t* part_empty = part_full + BUFS;              // [bufs] used in CTA 0: folds of both CTAs -> MMA
  uint64_t* sc_full = part_empty + BUFS;                // [slots] factor warps -> fold
  uint64_t* sc_empty = sc_full + SC_SLOTS;              // [slots] fold -> factor warps
  uint64_t* pair_bar = sc_empty + SC_SLOTS;             // [8] the two warps that exchange sums
  uint64_t* list_bars = pair_bar + 8;                   // [4] (PairList)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(list_bars + 4);
  int4* list = reinterpret_cast<int4*>(smem + STAGES * STAGE_BYTES + BAR_BYTES);
  uint8_t* strips = smem + STAGES * STAGE_BYTES + BAR_BYTES + kListBytes;
  uint8_t* factors = strips + kFoldWarps * G::STRIP_BYTES;                      // [slot][K block][gate | up][token]
  int32_t* meta = reinterpret_cast<int32_t*>(factors + G::FACTOR_BYTES);        // [tile][slot ids | row weights]
  uint8_t* exchange = factors + G::FACTOR_BYTES + G::META_BYTES;                 // [warp][round parity][4][lane] f32 pairs
  int32_t* table = reinterpret_cast<int32_t*>(exchange + kFoldWarps * G::EX_BYTES);

  const int warp = ptx::uniform_warp_id(), lane = threadIdx.x & 31;
  const int rank = (int)ptx::cluster_ctarank();
  const int worker = blockIdx.x >> 1, workers = gridDim.x >> 1;
  const long long t_kernel0 = PROF ? clock64() : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < BUFS; ++b) {
      ptx::mbar_init(&part_full[b], 1);
      ptx::mbar_init(&part_empty[b], kFoldWarps);  // the 8 warps of both CTAs that fold this K block
    }
    for (int s = 0; s < SC_SLOTS; ++s) {
      ptx::mbar_init(&sc_full[s], 1);
      ptx::mbar_init(&sc_empty[s], kFoldWarps);
    }
    for (int w = 0; w < 8; ++w) ptx::mbar_init(&pair_bar[w], 2);
    PairList::init_barriers(list_bars, kFoldWarps + 3 + (rank == 0));  // TMA, two factor warps, MMA
    ptx::fence_barrier_init();
  }
  if (warp == kFoldWarps && lane == 0) {
    ptx::prefetch_tensormap(&map_t);
    ptx::prefetch_tensormap(&map_w);
  }
  if (warp == kFoldWarps + 1) {
    ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  // behind a late trigger a given table is complete by now (see pdl_entry_late): only rows, scales and outputs wait
  const bool early = p.early;
  if (!early) pdl_wait();
  const int used_blocks = p.expert_table ? 0 : min((int)(*p.num_tokens_post_padded / 128), p.max_blocks);
  pair_build_table(table, p.num_experts, p.expert_table, p.expert_ids, p.sorted_token_ids, p.numel, 128, TOK,
                   used_blocks, p.min_rows, p.max_rows);
  ptx::cluster_sync_all();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int kblocks = p.kblocks;
  const int total_tiles = table[3 * p.num_experts] * p.w_tiles;
  PairList units(list, list_bars);
  PairUnit unit;
  const PairTile& tl = unit.tl;

  if (MOVE && warp >= kFoldWarps) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
  if (warp == kFoldWarps) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      const uint32_t ring = ptx::smem_u32(smem), bar_full0 = ptx::smem_u32(full_bar) & ~ptx::kPeerRankBit;
      for (bool first = true; alive; first = false) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x5c0);
          break;
        }
        const int half_n = tl.n >> 1;
        const int row_t = tl.row0 + rank * half_n;
        const int boxes = (half_n + BOX_TOKENS - 1) / BOX_TOKENS;
        const uint32_t bytes = 2 * (W_BYTES + boxes * (BOX_TOKENS * KBYTES));
        const int32_t c0 = GATED ? tl.w_tile * 128 + rank * 64 : tl.w_tile * 256 + rank * 128;
        auto load_weights = [&](int kb, int s) {  // arms the stage for the bytes of all its loads
          const uint32_t sw = ring + s * STAGE_BYTES, bar0 = bar_full0 + s * 8;
          const int32_t x = kb * KBYTES;  // element coordinate (1-byte elements)
          if (rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], bytes);
          if constexpr (GATED) ptx::tma_load_5d_pair(sw, &map_w, x, 0, 0, c0 >> 4, tl.expert, bar0);
          else ptx::tma_load_3d_pair(sw, &map_w, x, c0, tl.expert, bar0);
        };
        auto load_tokens = [&](int kb, int s) {
          for (int b = 0; b < boxes; ++b)
            ptx::tma_load_2d_pair(ring + s * STAGE_BYTES + W_BYTES + b * (BOX_TOKENS * KBYTES), &map_t, kb * KBYTES,
                                  row_t + b * BOX_TOKENS, bar_full0 + s * 8);
        };
        int kb = 0;
        if (first) {
          // the first tile's weights are on their way before the rows are there
          const int ahead = early ? min(STAGES, kblocks) : 0;
          for (; kb < ahead; ++kb) load_weights(kb, kb);
          pdl_wait();
          for (int s = 0; s < ahead; ++s) load_tokens(s, s);
          stage = ahead == STAGES ? 0 : ahead;
          phase = ahead == STAGES;
        }
        for (; kb < kblocks; ++kb) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report(0x500 | stage);
            alive = false;
            break;
          }
          load_weights(kb, stage);
          load_tokens(kb, stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (alive) {  // drain our own bulk copies before leaving
        for (int s = 0; s < STAGES; ++s) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report(0x580 | stage);
            break;
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == kFoldWarps + 1) {
    // ---------------- MMA issuer (CTA 0): one fresh partial per K block ----------------
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0, step = 0;  // step: K blocks issued so far (selects the partial and its phase)
      bool alive = true;
      long long prof_mp = 0, prof_md = 0;
      const uint32_t ring = ptx::smem_u32(smem);
      const uint64_t da0 = ptx::smem_desc_sw128(ring), db0 = ptx::smem_desc_sw128(ring + W_BYTES);
      while (alive) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x5d0);
          break;
        }
        const uint32_t idesc = ptx::make_idesc(/*e4m3*/ 0, 256, (uint32_t)tl.n);
        for (int kb = 0; kb < kblocks; ++kb, ++step) {
          const int buf = step % BUFS;
          const long long tm0 = PROF ? clock64() : 0;
          if (!ptx::mbar_wait(&part_empty[buf], ((step / BUFS) & 1) ^ 1)) {
            report(0x600 | buf);
            alive = false;
            break;
          }
          const long long tm1 = PROF ? clock64() : 0;
          if (!ptx::mbar_wait(&full_bar[stage], phase)) {
            report(0x640 | stage);
            alive = false;
            break;
          }
          if (PROF) {
            prof_mp += tm1 - tm0;
            prof_md += clock64() - tm1;
          }
          ptx::tc_fence_after_sync();
          const uint64_t da = da0 + (uint64_t)(stage * (STAGE_BYTES >> 4)), db = db0 + (uint64_t)(stage * (STAGE_BYTES >> 4));
          const uint32_t d_tmem = tmem_base + buf * TOK;
#pragma unroll
          for (int kk = 0; kk < KBYTES / 32; ++kk)
            ptx::mma_f8f6f4_ss_pair(d_tmem, da + 2 * kk, db + 2 * kk, idesc, kk != 0);
          ptx::mma_commit_both(&part_full[buf]);
          ptx::mma_commit_both(&empty_bar[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (PROF && blockIdx.x < 256) {
        g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 6] = prof_mp;
        g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 7] = prof_md;
      }
    }
  } else if (warp >= kFoldWarps + 2) {
    // ---------------- factors: two warps take alternate groups of four K blocks, one tile after the other ----------------
    constexpr int LANES = TOK / 32;  // tokens per lane
    const int me = warp - (kFoldWarps + 2);
    int more = 0;  // the list goes on
    auto add_units = [&](int batch) {
      more = PairList::fill(list, list_bars, batch, worker, workers, total_tiles, p.w_tiles, p.group, p.num_experts, table);
      if (more < 0) report(0x5b0);
    };
    if (me == 0) add_units(0);
    pdl_wait();
    uint32_t group = 0;  // groups so far (selects the slot and its phase)
    bool alive = true;
    int ltile = 0;
    const bool vec = (kblocks & 3) == 0 && aligned16(p.a_scale) && aligned16(p.w_scale);
    const int wblocks = (int)(p.w_rows / 128);
    for (; alive; ++ltile) {
      // half a batch ahead: every reader is at most a few tiles (of the factor ring) behind, so nobody is waited for
      if (more > 0 && ltile % kListUnits == kListUnits / 2) add_units(ltile / kListUnits + 1);
      const int got = units.next<true>(&unit);
      if (got <= 0) {
        if (got < 0) report(0x5e0);
        break;
      }
      int32_t ids[LANES], row[LANES];  // slot and scale row of token lane + 32 j
#pragma unroll
      for (int j = 0; j < LANES; ++j) {
        const int u = lane + 32 * j;
        ids[j] = u < tl.cols ? p.sorted_token_ids[tl.row0 + u] : -1;
      }
#pragma unroll
      for (int j = 0; j < LANES; ++j) {
        if (ids[j] >= p.numel) ids[j] = -1;
        row[j] = ids[j] < 0 ? 0 : (p.a_scale_gather ? ids[j] / p.top_k : tl.row0 + lane + 32 * j);
      }
      const int w0 = GATED ? tl.w_tile : min(tl.w_tile * 2 + rank, wblocks - 1), w1 = GATED ? tl.w_tile + wblocks / 2 : w0;
      const float* sw0 = p.w_scale + ((int64_t)tl.expert * wblocks + w0) * kblocks;
      const float* sw1 = p.w_scale + ((int64_t)tl.expert * wblocks + w1) * kblocks;
      for (int kb0 = 0; kb0 < kblocks; kb0 += 4, ++group) {
        if ((int)(group & 1) != me) continue;
        float4 a[LANES], f0, f1;
        if (vec) {
          f0 = __ldg(reinterpret_cast<const float4*>(sw0 + kb0));
          f1 = GATED ? __ldg(reinterpret_cast<const float4*>(sw1 + kb0)) : f0;
#pragma unroll
          for (int j = 0; j < LANES; ++j)  // a tile's unused lanes read row 0 and store factors that nobody uses
            if (32 * j < tl.n) a[j] = __ldg(reinterpret_cast<const float4*>(p.a_scale + (int64_t)row[j] * kblocks + kb0));
        } else {
          const int left = kblocks - kb0;
          auto load4 = [&](const float* src) {
            return make_float4(src[0], left > 1 ? src[1] : 0.f, left > 2 ? src[2] : 0.f, left > 3 ? src[3] : 0.f);
          };
          f0 = load4(sw0 + kb0);
          f1 = GATED ? load4(sw1 + kb0) : f0;
#pragma unroll
          for (int j = 0; j < LANES; ++j)
            if (32 * j < tl.n) a[j] = load4(p.a_scale + (int64_t)row[j] * kblocks + kb0);
        }
        const int slot = group % SC_SLOTS;
        if (!warp_wait(&sc_empty[slot], ((group / SC_SLOTS) & 1) ^ 1)) {
          report(0x780 | slot);
          alive = false;
          break;
        }
        if constexpr (!GATED) {
          if (kb0 == 0) {  // the slot just granted also frees this tile's meta entry
            int32_t* m = meta + (ltile % META_TILES) * TOK * 2;
#pragma unroll
            for (int j = 0; j < LANES; ++j) {
              m[lane + 32 * j] = ids[j];
              m[TOK + lane + 32 * j] = __float_as_int((ids[j] >= 0 && p.row_scale) ? p.row_scale[ids[j]] : 1.0f);
            }
          }
        }
        float* dst = reinterpret_cast<float*>(factors + slot * 4 * KB_BYTES) + lane;
        constexpr int KB_STEP = KB_BYTES / 4;
#pragma unroll
        for (int j = 0; j < LANES; ++j) {
          if (32 * j < tl.n) {
            float* d = dst + 32 * j;
            d[0] = a[j].x * f0.x;
            d[KB_STEP] = a[j].y * f0.y;
            d[2 * KB_STEP] = a[j].z * f0.z;
            d[3 * KB_STEP] = a[j].w * f0.w;
            if constexpr (GATED) {
              d[TOK] = a[j].x * f1.x;
              d[KB_STEP + TOK] = a[j].y * f1.y;
              d[2 * KB_STEP + TOK] = a[j].z * f1.z;
              d[3 * KB_STEP + TOK] = a[j].w * f1.w;
            }
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sc_full[slot]);
      }
    }
  } else {
    // ---------------- fold + epilogue (warps 0-15) ----------------
    if constexpr (MOVE) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFoldRegs));
    pdl_entry_late();
    const int quarter = warp & 3, half = (warp >> 2) & 1, kgroup = warp >> 3;
    const int t = lane & 3;
    const uint32_t factor_addr = ptx::smem_u32(factors) + (16 * half + 2 * t) * 4;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + 16 * half;
    const uint32_t full0 = ptx::smem_u32(part_full), to_empty = BUFS * 8;  // part_empty follows part_full
    const uint32_t out_addr = ptx::smem_u32(exchange) + warp * G::EX_BYTES + lane * 8;
    const uint32_t in_addr = ptx::smem_u32(exchange) + (warp ^ 8) * G::EX_BYTES + lane * 8;
    uint32_t step0 = 0, slot = 0;  // K blocks before this tile; factor slots used
    int ltile = 0;
    bool alive = true;
    long long prof_fw = 0, prof_fb = 0, prof_sw = 0, prof_epi = 0;
    for (; alive; ++ltile) {
      const int got = units.next<true>(&unit);
      if (got <= 0) {
        if (got < 0) report(0x5f0);
        break;
      }
      const int pieces = max(0, ((tl.n >> 4) - half + 1) >> 1);  // 16-token pieces half, half + 2, ..
      unsigned long long acc[PIECES][8];  // [0..3] rows 0-15 of the quarter, [4..7] rows 16-31
#pragma unroll
      for (int q = 0; q < 8 * PIECES; ++q) acc[q / 8][q % 8] = 0ull;
#pragma unroll 1
      for (int kb0 = 0; kb0 < kblocks; kb0 += 4, ++slot) {
        const long long tf0 = PROF ? clock64() : 0;
        if (!warp_wait(&sc_full[slot % SC_SLOTS], (slot / SC_SLOTS) & 1)) {
          report(0x740);
          alive = false;
          break;
        }
        if (PROF) prof_sw += clock64() - tf0;
        // the K blocks with this group's parity, counted over all tiles: a partial then always belongs to the same group
#pragma unroll 1
        for (int kb = kb0 + (int)((kgroup ^ (step0 + kb0)) & 1); kb < min(kb0 + 4, kblocks); kb += 2) {
          const uint32_t step = step0 + kb, buf = step % BUFS;
          const long long tf1 = PROF ? clock64() : 0;
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_addr(full0 + buf * 8, (step / BUFS) & 1))) {
            report(0x700);
            alive = false;
            break;
          }
          const long long tf2 = PROF ? clock64() : 0;
          ptx::tc_fence_after_sync();
          const uint32_t taddr = lane_addr + buf * TOK;
          const uint32_t fsrc = factor_addr + ((slot % SC_SLOTS) * 4 + (kb - kb0)) * KB_BYTES;
          auto hand_back = [&]() {  // the partial is in registers
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (ptx::elect_one()) ptx::mbar_arrive_cluster(((full0 + buf * 8) & ~ptx::kPeerRankBit) + to_empty);
          };
          if (pieces > 0) {
            uint32_t lo[PIECES][8], hi[PIECES][8];
            unsigned long long g[PIECES][2], u[PIECES][2];
#pragma unroll
            for (int q = 0; q < PIECES; ++q) {  // columns past the tile's tokens hold leftovers that nobody stores
              ptx::tmem_ld_16x256b_x2(taddr + 32 * q, lo[q]);
              ptx::tmem_ld_16x256b_x2(taddr + 32 * q + (16u << 16), hi[q]);
              g[q][0] = lds64(fsrc + 128 * q);
              g[q][1] = lds64(fsrc + 128 * q + 32);
              u[q][0] = GATED ? lds64(fsrc + 128 * q + TOK * 4) : g[q][0];
              u[q][1] = GATED ? lds64(fsrc + 128 * q + TOK * 4 + 32) : g[q][1];
            }
            ptx::tmem_ld_wait();
            hand_back();
#pragma unroll
            for (int q = 0; q < PIECES; ++q) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                fma2(acc[q][c], lo[q][2 * c], lo[q][2 * c + 1], g[q][c >> 1]);
                fma2(acc[q][4 + c], hi[q][2 * c], hi[q][2 * c + 1], u[q][c >> 1]);
              }
            }
          } else {
            hand_back();
          }
          if (PROF) {
            prof_fw += tf2 - tf1;
            prof_fb += clock64() - tf2;
          }
        }
        if (!alive) break;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sc_empty[slot % SC_SLOTS]);
      }
      step0 += kblocks;
      if (!alive) break;

      const long long te0 = PROF ? clock64() : 0;
      const int32_t* m = meta + (ltile % META_TILES) * TOK * 2;
      uint8_t* strip = strips + warp * G::STRIP_BYTES;
      const int ch0 = GATED ? tl.w_tile * 128 + rank * 64 + quarter * 16 : tl.w_tile * 256 + rank * 128 + quarter * 32;
      // The two K groups' sums meet: each warp hands one piece to its partner (same channels and tokens, other group) and
      // finishes the other.  Two rounds, two buffers: the partner has read one before it arrives for the next.
      if (pieces > 0) {
        unsigned long long sum[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int c = 0; c < 4; ++c) sts64(out_addr + h * 1024 + c * 256, kgroup ? acc[0][4 * h + c] : acc[1][4 * h + c]);
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&pair_bar[warp & 7]);
          if (!warp_wait(&pair_bar[warp & 7], h)) {  // two rounds per tile: h is the phase
            report(0x7c0);
            alive = false;
          }
#pragma unroll
          for (int c = 0; c < 4; ++c)
            sum[4 * h + c] = add2(kgroup ? acc[1][4 * h + c] : acc[0][4 * h + c], lds64(in_addr + h * 1024 + c * 256));
        }
        if (!alive) break;
        if (kgroup < pieces) {
          const int tok0 = 16 * half + 32 * kgroup;
          float2 r0 = make_float2(1.f, 1.f), r1 = r0;
          if constexpr (!GATED) {
            r0 = *reinterpret_cast<const float2*>(m + TOK + tok0 + 2 * t);
            r1 = *reinterpret_cast<const float2*>(m + TOK + tok0 + 8 + 2 * t);
          } else if (p.row_scale) {  // top-k weight on the input side: not the usual case, looked up in place
            r0 = make_float2(row_weight(p, tl, tok0 + 2 * t), row_weight(p, tl, tok0 + 2 * t + 1));
            r1 = make_float2(row_weight(p, tl, tok0 + 8 + 2 * t), row_weight(p, tl, tok0 + 9 + 2 * t));
          }
          float lo[8], hi[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            unpack2(sum[q], lo[2 * q], lo[2 * q + 1]);
            unpack2(sum[4 + q], hi[2 * q], hi[2 * q + 1]);
          }
          const float rs[4] = {r0.x, r0.y, r1.x, r1.y};
          if constexpr (GATED) {
            // element j: token tok0 + 8 * (j >> 2) + 2 t + (j & 1), channel ch0 + lane / 4 + 8 * ((j >> 1) & 1)
#pragma unroll
            for (int j = 0; j < 8; ++j) lo[j] = act_mul(lo[j] * rs[2 * (j >> 2) + (j & 1)], hi[j] * rs[2 * (j >> 2) + (j & 1)], p.activation);
            if (p.out_dtype == FMOE_F32) {  // eight lanes store one token's 32 bytes
              const int row0 = p.by_expert ? tl.row0 - table[tl.expert] + tl.expert * kNarrowRows : tl.row0;
              float* out = reinterpret_cast<float*>(p.out) + (int64_t)(row0 + tok0) * p.n + ch0 + (lane >> 2);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int u = 8 * (j >> 2) + 2 * t + (j & 1);
                if (u < tl.cols - tok0) out[(int64_t)u * p.n + 8 * ((j >> 1) & 1)] = lo[j];
              }
            } else {
              uint32_t v[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) v[q] = pack_bf16x2(lo[2 * q], lo[2 * q + 1]);
              strip_put16(strip, 48, 0, lane, v);
              strip_store_sorted(strip, lane, reinterpret_cast<__nv_bfloat16*>(p.out) + (int64_t)(tl.row0 + tok0) * p.n, p.n, ch0,
                                 tl.cols - tok0);
            }
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t v[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int j = 4 * (q >> 1) + 2 * (q & 1);
                const float a0 = h ? hi[j] : lo[j], a1 = h ? hi[j + 1] : lo[j + 1];
                v[q] = pack_bf16x2(a0 * rs[2 * (q >> 1)], a1 * rs[2 * (q >> 1) + 1]);
              }
              strip_put16(strip, 80, 16 * h, lane, v);
            }
            strip_store_slots(strip, lane, p.out, p.out_rows, p.n, ch0, m[tok0 + (lane >> 2)], m[tok0 + 8 + (lane >> 2)]);
          }
        }
      }
      if constexpr (GATED) {
        if (p.zero_padding && tl.last)
          zero_block_rows(tl, p.out, p.n, tl.w_tile * 128 + rank * 64, p.out_dtype == FMOE_F32 ? 4 : 2, threadIdx.x, kFoldWarps * 32);
      }
      if (PROF) prof_epi += clock64() - te0;
    }
    if (p.out_rows) __threadfence_system();  // rows stored to a peer are complete before the kernel ends
    if (PROF && threadIdx.x == 0 && blockIdx.x < 256) {
      long long* out = g_wait_prof_fp8 + (GATED ? 2048 : 0) + blockIdx.x * 8;
      out[0] = ltile;
      out[1] = prof_fw;
      out[2] = prof_fb;
      out[3] = prof_sw;
      out[4] = prof_epi;
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();  // nobody signals into a CTA that has left, and both are done with TMEM
  if (warp == kFoldWarps + 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  if (PROF && threadIdx.x == 0 && blockIdx.x < 256)
    g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 5] = clock64() - t_kernel0;
}

// ---------------------------------------------------------------------------------------------------------------------
// Wide tiles (experts with many rows): the same fold with the TOKENS on the M side, up to 256 of one expert (128 in each CTA)
// x 256 weight rows (CTA 0 loads the tile's first 64 gate and 64 up channels, in turns of 16, or its first 128 rows; CTA 1
// the others).  A thread of the fold then owns one token: its activation scale is ONE value per K block and the weight scale
// one value per 128 rows, and TMEM is read 32 lanes wide (136 cycles for a 128 x 256 partial, its FMAs 256).  With tokens on N
// every thread needs one factor per column: a 16-lane read-out with packed factors takes 128-256 shared-memory loads per
// partial, a 32-lane one 1024 cycles of broadcast loads, against 32 loads here.
//   M = 256, or 128 where the tile has at most 128 tokens (an expert's last or only tile: all others have 256).  An MMA of
//   M = 128 takes as long, but leaves half as much to fold, half the lanes' power unspent and a third of shared memory's
//   traffic: 0.50 us per K block and tile against 0.66 (DeepSeek-V3, 64 experts of 128 rows, both GEMMs: 717 -> 610 us; as
//   M = 256 with lanes to spare such a tile took as long as a full one).  Its layout: lanes 0-63 hold the CTA's 64 tokens x
//   CTA 0's weight rows, lanes 64-127 the same tokens x CTA 1's.
//   TMEM: four partials of 128 columns (M = 128: the first 64 of each).  A K block's MMAs go to two of them: the first holds
//   rows 0-63 of both CTAs' weights, the second rows 64-127.
//   warps 0-15: fold + epilogue.  Eight warps fold each half, so that one half's TMEM reads run beside the other's FMAs and a
//   partial is handed back while the other half is still being multiplied (one partial of 256 columns per K block, folded by
//   all sixteen warps at once: gate/up + down of DeepSeek-V3, 4096 tokens, 3.43 ms; this split 3.25 ms).  Warp w: TMEM lanes
//   32 * (w % 4).., half w / 8, the 64 columns of CTA w / 4 % 2's weight rows (M = 128: 32 columns): 64 accumulators per
//   thread.  (Eight warps with 128 accumulators each spill: 530 -> 700 us and more.)
//   warp 16 TMA, warp 17 MMA (CTA 0), warps 18-19 factors: products of token and weight scales in a ring of 4 slots of 8 K
//   blocks, one slot wait per 8 K blocks of the fold.  What would not fit their 64 registers is left out of their loop: it is not
//   unrolled over the slot's halves (gate/up GEMM, 256 rows, 545 us with it, 519 without), and the path for scales that 16-byte
//   loads cannot take is a kernel of its own (VEC; with both in one, and the epilogue as it was, 116 and 88 bytes were
//   loaded back: DeepSeek-V3, 4096 tokens, 3150 -> 2985 us without, 1024 1680 -> 1633, 16384 8913 -> 8362).  The fold warps' 104
//   registers hold the epilogue because the activation is chosen once for a tile, not per value.
// The gate/up kernel quantises its output: the tile's 128 channels of a token are one group, spread over four warps (M = 128:
// eight), which exchange their largest magnitudes through shared memory.  (A bf16 activation and a quantiser pass took 135 us
// of that case.)
// What bounds it: shared memory (M = 256: 32 KB in and 48 KB of operand reads per K block, 640 cycles; the fold's round trip
// through two partials makes it about 800), at the SM clock that the power limit leaves (1.4 GHz of 1.965).
// ---------------------------------------------------------------------------------------------------------------------
struct WideGeo {
  static constexpr int STAGE_BYTES = 2 * W_BYTES;  // 128 token rows + 128 weight rows per CTA
  static constexpr int STAGES = 5;
  static constexpr int GROUP = 8;                  // K blocks per factor slot
  static constexpr int KB_BYTES = 2 * 128 * 4;     // factors of one K block: [first | second 128 columns][token]
  static constexpr int SLOT_BYTES = GROUP * KB_BYTES;
  static constexpr int META_WORDS = 2 * 128 + 4;   // slot ids, row weights, {first row, rows of this CTA, weight tile}
  static constexpr int META_BYTES = META_TILES * META_WORDS * 4;
  // two tiles' [column piece][token] largest magnitudes: four pieces of 128 tokens, then eight of 64 (M = 128)
  static constexpr int AMAX_BYTES = 2 * (4 * 128 + 8 * 64) * 4;
  static constexpr int bytes(int num_experts) {
    return STAGES * STAGE_BYTES + BAR_BYTES + kListBytes + SC_SLOTS * SLOT_BYTES + META_BYTES + AMAX_BYTES + pair_table_bytes(num_experts);
  }
};
static_assert(WideGeo::bytes(1024) <= kMaxSmem, "shared memory");

// VEC: the scales of four K blocks are one 16-byte load
template <bool GATED, bool PROF, bool MOVE, bool VEC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
grouped_gemm_pair_fold_wide_kernel(const __grid_constant__ CUtensorMap map_t, const __grid_constant__ CUtensorMap map_w,
                                   const FoldParams p) {
  using G = WideGeo;
  constexpr int STAGES = G::STAGES, STAGE_BYTES = G::STAGE_BYTES;
  extern __shared__ __align__(1024) uint8_t smem[];  // aligned by declaration: every address below is a constant
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full_bar = bars;                 // [STAGES] used in CTA 0: both CTAs' loads -> MMA
  uint64_t* empty_bar = bars + STAGES;       // [STAGES] per CTA: MMA -> producer
  uint64_t* part_full = bars + 2 * STAGES;   // [4] per CTA: MMA -> fold
  uint64_t* part_empty = part_full + 4;      // [4] used in CTA 0: folds of both CTAs -> MMA
  uint64_t* sc_full = part_empty + 4;        // [slots] scale warps -> fold
  uint64_t* sc_empty = sc_full + SC_SLOTS;   // [slots] fold -> scale warps
  uint64_t* amax_bar = sc_empty + SC_SLOTS;  // [4] the four warps that hold a token's 128 channels
  uint64_t* small_bar = amax_bar + 4;        // [2] M = 128: the eight warps that hold a token's 128 channels
  uint64_t* list_bars = small_bar + 2;       // [4] (PairList)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(list_bars + 4);
  int4* list = reinterpret_cast<int4*>(smem + STAGES * STAGE_BYTES + BAR_BYTES);
  uint8_t* scales = smem + STAGES * STAGE_BYTES + BAR_BYTES + kListBytes;  // [slot][K block][half][token]
  int32_t* meta = reinterpret_cast<int32_t*>(scales + SC_SLOTS * G::SLOT_BYTES);  // [tile]
  float* amax_buf = reinterpret_cast<float*>(scales + SC_SLOTS * G::SLOT_BYTES + G::META_BYTES);
  int32_t* table = reinterpret_cast<int32_t*>(scales + SC_SLOTS * G::SLOT_BYTES + G::META_BYTES + G::AMAX_BYTES);

  const int warp = ptx::uniform_warp_id(), lane = threadIdx.x & 31;
  const int rank = (int)ptx::cluster_ctarank();
  const int worker = blockIdx.x >> 1, workers = gridDim.x >> 1;
  const long long t_kernel0 = PROF ? clock64() : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 4; ++b) {
      ptx::mbar_init(&part_full[b], 1);
      ptx::mbar_init(&part_empty[b], kFoldWarps);  // the half's 8 warps of both CTAs
      ptx::mbar_init(&amax_bar[b], 4);
    }
    for (int s = 0; s < SC_SLOTS; ++s) {
      ptx::mbar_init(&sc_full[s], 1);
      ptx::mbar_init(&sc_empty[s], kFoldWarps);
    }
    for (int b = 0; b < 2; ++b) ptx::mbar_init(&small_bar[b], 8);
    PairList::init_barriers(list_bars, 3 + (rank == 0));  // TMA, two factor warps, MMA
    ptx::fence_barrier_init();
  }
  if (warp == kFoldWarps && lane == 0) {
    ptx::prefetch_tensormap(&map_t);
    ptx::prefetch_tensormap(&map_w);
  }
  if (warp == kFoldWarps + 1) {
    ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  const bool early = p.early;
  if (!early) pdl_wait();
  const int used_blocks = p.expert_table ? 0 : min((int)(*p.num_tokens_post_padded / 128), p.max_blocks);
  pair_build_table(table, p.num_experts, p.expert_table, p.expert_ids, p.sorted_token_ids, p.numel, 128, 256, used_blocks,
                   p.min_rows, p.max_rows);
  ptx::cluster_sync_all();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int kblocks = p.kblocks;
  const int total_tiles = table[3 * p.num_experts] * p.w_tiles;
  PairList units(list, list_bars);
  PairUnit unit;
  const PairTile& tl = unit.tl;

  if (MOVE && warp >= kFoldWarps) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
  if (warp == kFoldWarps) {
    // ---------------- TMA producer (both CTAs): its half of the tile's tokens, its 128 weight rows ----------------
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      const uint32_t ring = ptx::smem_u32(smem), bar_full0 = ptx::smem_u32(full_bar) & ~ptx::kPeerRankBit;
      for (bool first = true; alive; first = false) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x5c0);
          break;
        }
        const int half_n = tl.n >> 1;
        const int row_t = tl.row0 + rank * half_n;
        const int boxes = (half_n + BOX_TOKENS - 1) / BOX_TOKENS;  // lanes past them multiply what an earlier stage left
        const uint32_t bytes = 2 * (W_BYTES + boxes * (BOX_TOKENS * KBYTES));
        const int32_t c0 = GATED ? tl.w_tile * 128 + rank * 64 : tl.w_tile * 256 + rank * 128;
        auto load_weights = [&](int kb, int s) {
          const uint32_t sw = ring + s * STAGE_BYTES + W_BYTES, bar0 = bar_full0 + s * 8;
          if (rank == 0) ptx::mbar_arrive_expect_tx(&full_bar[s], bytes);
          if constexpr (GATED) ptx::tma_load_5d_pair(sw, &map_w, kb * KBYTES, 0, 0, c0 >> 4, tl.expert, bar0);
          else ptx::tma_load_3d_pair(sw, &map_w, kb * KBYTES, c0, tl.expert, bar0);
        };
        auto load_tokens = [&](int kb, int s) {
          for (int b = 0; b < boxes; ++b)
            ptx::tma_load_2d_pair(ring + s * STAGE_BYTES + b * (BOX_TOKENS * KBYTES), &map_t, kb * KBYTES, row_t + b * BOX_TOKENS,
                                  bar_full0 + s * 8);
        };
        int kb = 0;
        if (first) {
          // the first tile's weights are on their way before the rows are there
          const int ahead = early ? min(STAGES, kblocks) : 0;
          for (; kb < ahead; ++kb) load_weights(kb, kb);
          pdl_wait();
          for (int s = 0; s < ahead; ++s) load_tokens(s, s);
          stage = ahead == STAGES ? 0 : ahead;
          phase = ahead == STAGES;
        }
        for (; kb < kblocks; ++kb) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report(0x500 | stage);
            alive = false;
            break;
          }
          load_weights(kb, stage);
          load_tokens(kb, stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (alive) {
        for (int s = 0; s < STAGES; ++s) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report(0x580 | stage);
            break;
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == kFoldWarps + 1) {
    // ---------------- MMA issuer (CTA 0): one fresh partial per K block ----------------
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0, step = 0;
      bool alive = true;
      long long prof_mp = 0, prof_md = 0;
      const uint32_t ring = ptx::smem_u32(smem);
      const uint64_t da0 = ptx::smem_desc_sw128(ring), db0 = ptx::smem_desc_sw128(ring + W_BYTES);
      while (alive) {
        const int got = units.next<false>(&unit);
        if (got <= 0) {
          if (got < 0) report(0x5d0);
          break;
        }
        const uint32_t idesc = ptx::make_idesc(/*e4m3*/ 0, tl.n <= 128 ? 128 : 256, 128);
        for (int kb = 0; kb < kblocks; ++kb, ++step) {
          const long long tm0 = PROF ? clock64() : 0;
          if (!ptx::mbar_wait(&full_bar[stage], phase)) {  // the data is there long before the partial is folded
            report(0x640 | stage);
            alive = false;
            break;
          }
          if (PROF) prof_md += clock64() - tm0;
          const uint64_t da = da0 + (uint64_t)(stage * (STAGE_BYTES >> 4)), db = db0 + (uint64_t)(stage * (STAGE_BYTES >> 4));
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // half h: rows 64 h.. of both CTAs' weight rows
            const int buf = 2 * (step & 1) + h;
            const long long tm1 = PROF ? clock64() : 0;
            if (!ptx::mbar_wait(&part_empty[buf], ((step >> 1) & 1) ^ 1)) {
              report(0x600 | buf);
              alive = false;
              break;
            }
            if (PROF) prof_mp += clock64() - tm1;
            ptx::tc_fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < KBYTES / 32; ++kk)
              ptx::mma_f8f6f4_ss_pair(tmem_base + buf * 128, da + 2 * kk, db + h * (64 * KBYTES >> 4) + 2 * kk, idesc, kk != 0);
            ptx::mma_commit_both(&part_full[buf]);
          }
          if (!alive) break;
          ptx::mma_commit_both(&empty_bar[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (PROF && blockIdx.x < 256) {
        g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 6] = prof_mp;
        g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 7] = prof_md;
      }
    }
  } else if (warp >= kFoldWarps + 2) {
    // ---------------- factors: two warps take alternate groups of eight K blocks ----------------
    const int me = warp - (kFoldWarps + 2);
    int more = 0;
    auto add_units = [&](int batch) {
      more = PairList::fill(list, list_bars, batch, worker, workers, total_tiles, p.w_tiles, p.group, p.num_experts, table, 256);
      if (more < 0) report(0x5b0);
    };
    if (me == 0) add_units(0);
    pdl_wait();
    uint32_t group = 0;
    bool alive = true;
    int ltile = 0;
    const int wblocks = (int)(p.w_rows / 128);
    for (; alive; ++ltile) {
      // half a batch ahead: every reader is at most a few tiles (of the factor ring) behind, so nobody is waited for
      if (more > 0 && ltile % kListUnits == kListUnits / 2) add_units(ltile / kListUnits + 1);
      const int got = units.next<true>(&unit);
      if (got <= 0) {
        if (got < 0) report(0x5e0);
        break;
      }
      const int half_n = tl.n >> 1, first = tl.row0 + rank * half_n;
      int32_t ids[4], row[4];  // slot and scale row of this CTA's token lane + 32 j
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int u = lane + 32 * j;
        ids[j] = (u < half_n && rank * half_n + u < tl.cols) ? p.sorted_token_ids[first + u] : -1;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (ids[j] >= p.numel) ids[j] = -1;
        row[j] = ids[j] < 0 ? 0 : (p.a_scale_gather ? ids[j] / p.top_k : first + lane + 32 * j);
      }
      const int w0 = GATED ? tl.w_tile : tl.w_tile * 2, w1 = GATED ? tl.w_tile + wblocks / 2 : min(tl.w_tile * 2 + 1, wblocks - 1);
      const float* sw0 = p.w_scale + ((int64_t)tl.expert * wblocks + w0) * kblocks;
      const float* sw1 = p.w_scale + ((int64_t)tl.expert * wblocks + w1) * kblocks;
      for (int kb0 = 0; kb0 < kblocks; kb0 += G::GROUP, ++group) {
        if ((int)(group & 1) != me) continue;
        const int slot = group % SC_SLOTS;
        bool granted = false;
#pragma unroll 1
        for (int q = 0; q < G::GROUP / 4; ++q) {
          const int kb = kb0 + 4 * q, left = kblocks - kb;
          if (left <= 0) break;
          float4 a[4], f0, f1;
          if constexpr (VEC) {
            f0 = __ldg(reinterpret_cast<const float4*>(sw0 + kb));
            f1 = __ldg(reinterpret_cast<const float4*>(sw1 + kb));
#pragma unroll
            for (int j = 0; j < 4; ++j)  // tokens that are not there read row 0
              if (32 * j < half_n) a[j] = __ldg(reinterpret_cast<const float4*>(p.a_scale + (int64_t)row[j] * kblocks + kb));
          } else {
            auto load4 = [&](const float* src) {
              return make_float4(src[0], left > 1 ? src[1] : 0.f, left > 2 ? src[2] : 0.f, left > 3 ? src[3] : 0.f);
            };
            f0 = load4(sw0 + kb);
            f1 = load4(sw1 + kb);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (32 * j < half_n) a[j] = load4(p.a_scale + (int64_t)row[j] * kblocks + kb);
          }
          if (!granted) {
            if (!warp_wait(&sc_empty[slot], ((group / SC_SLOTS) & 1) ^ 1)) {
              report(0x780 | slot);
              alive = false;
              break;
            }
            granted = true;
            if (kb0 == 0) {  // the slot just granted also frees this tile's meta entry
              int32_t* m = meta + (ltile % META_TILES) * G::META_WORDS;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                m[lane + 32 * j] = ids[j];
                m[128 + lane + 32 * j] = __float_as_int((ids[j] >= 0 && p.row_scale) ? p.row_scale[ids[j]] : 1.0f);
              }
              if (lane == 0) {
                m[256] = first;
                m[257] = half_n;
                m[258] = tl.w_tile;
              }
            }
          }
          float* dst = reinterpret_cast<float*>(scales + slot * G::SLOT_BYTES + 4 * q * G::KB_BYTES) + lane;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (32 * j < half_n) {
              float* d = dst + 32 * j;
              d[0] = a[j].x * f0.x;
              d[128] = a[j].x * f1.x;
              d[256] = a[j].y * f0.y;
              d[384] = a[j].y * f1.y;
              d[512] = a[j].z * f0.z;
              d[640] = a[j].z * f1.z;
              d[768] = a[j].w * f0.w;
              d[896] = a[j].w * f1.w;
            }
          }
        }
        if (!alive) break;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sc_full[slot]);
      }
      if constexpr (GATED) {
        if (p.zero_padding && tl.last && me == 0) {  // rows between the expert's last token and its block's end
          zero_block_rows(tl, p.out, p.n, tl.w_tile * 128 + rank * 64,
                          p.out_dtype == FMOE_F32 ? 4 : (p.out_dtype == FMOE_BF16 ? 2 : 1), lane, 32);
        }
      }
    }
  } else {
    // ---------------- fold + epilogue (warps 0-15) ----------------
    if constexpr (MOVE) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFoldRegs));
    pdl_entry_late();
    // This loop runs at 104 registers (96 where the move is left out): the tile is described by its meta entry, shared
    // memory addresses are constants, everything else is derived from three counters.
    const uint32_t my_full = ptx::smem_u32(part_full) + 8 * (warp >> 3);  // the warp's half of the even K blocks
    constexpr uint32_t kToEmpty = 4 * 8;                                   // from part_full to part_empty
    uint32_t step = 0, group = 0;  // K blocks folded so far; factor slots used
    int ltile = 0;
    int small_tiles = 0;  // of them: the barriers of the two kinds of quantisation group have phases of their own
    bool alive = true;
    long long prof_fw = 0, prof_fb = 0, prof_sw = 0, prof_epi = 0;
    const volatile int32_t* tiles = table + 3 * p.num_experts;
    for (; worker + ltile * workers < *tiles * p.w_tiles; ++ltile) {
      // Gate/up: 16 gate channels, the same 16 of up, and 16 further of both; down: 64 channels (M = 128: the first half)
      float acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0.f;
      bool mine = false;   // some of this warp's lanes hold tokens
      bool small = false;  // M = 128: lanes 0-63 hold this CTA's 64 tokens x CTA 0's weight rows, lanes 64-127 x CTA 1's
      const int piece = (warp >> 2) & 1;
#pragma unroll 1
      for (int left = kblocks; left > 0; left -= G::GROUP, ++group) {
        const long long tf0 = PROF ? clock64() : 0;
        if (!warp_wait(&sc_full[group % SC_SLOTS], (group / SC_SLOTS) & 1)) {
          report(0x740);
          alive = false;
          break;
        }
        if (PROF) prof_sw += clock64() - tf0;
        const int tokens = meta[(ltile % META_TILES) * G::META_WORDS + 257];
        small = tokens <= 64;
        mine = (small ? warp & 1 : warp & 3) * 32 < tokens;
        uint32_t src = ptx::smem_u32(scales) + (group % SC_SLOTS) * G::SLOT_BYTES + ((small ? warp & 1 : warp & 3) * 32 + lane) * 4;
        if constexpr (!GATED) src += 512 * (small ? (warp >> 1) & 1 : piece);
        const uint32_t from = *reinterpret_cast<volatile uint32_t*>(tmem_slot) + ((uint32_t)((warp & 3) * 32) << 16) + 128 * (warp >> 3) +
                              (small ? 32 : 64) * piece;
        const uint32_t end = step + min(left, G::GROUP);
        // 16 columns at a time keeps the staging registers few (the 64 accumulators stay live)
        auto fold = [&](auto chunks_c) {
          constexpr int CHUNKS = decltype(chunks_c)::value;
#pragma unroll 1
          for (; step != end; ++step, src += G::KB_BYTES) {
            const uint32_t odd = step & 1;
            const long long tf1 = PROF ? clock64() : 0;
            if (!__all_sync(0xffffffffu, ptx::mbar_wait_addr(my_full + odd * 16, (step >> 1) & 1))) {
              report(0x700);
              alive = false;
              break;
            }
            const long long tf2 = PROF ? clock64() : 0;
            ptx::tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
              const float f = lds32(src + (GATED ? (c & 1) * 512 : 0));
              uint32_t v[16];
              ptx::tmem_ld_32x32b_x16(from + odd * 256 + c * 16, v);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[16 * c + i] = fmaf(__uint_as_float(v[i]), f, acc[16 * c + i]);
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (ptx::elect_one()) ptx::mbar_arrive_cluster(((my_full + odd * 16) & ~ptx::kPeerRankBit) + kToEmpty);
            if (PROF) {
              prof_fw += tf2 - tf1;
              prof_fb += clock64() - tf2;
            }
          }
        };
        if (!mine) fold(std::integral_constant<int, 0>{});
        else if (small) fold(std::integral_constant<int, 2>{});
        else fold(std::integral_constant<int, 4>{});
        if (!alive) break;
        if (lane == 0) ptx::mbar_arrive(&sc_empty[group % SC_SLOTS]);
      }
      if (!alive) break;

      const long long te0 = PROF ? clock64() : 0;
      const int32_t* m = meta + (ltile % META_TILES) * G::META_WORDS;
      const int tok = (small ? warp & 1 : warp & 3) * 32 + lane, half = warp >> 3;
      const int32_t slot = m[tok];
      const float rs = __int_as_float(m[128 + tok]);
      const int side = small ? (warp >> 1) & 1 : piece;  // whose weight rows: CTA 0's or CTA 1's
      if constexpr (GATED) {
        // output channels of the tile: 16 or 32 from here, in place of the gate accumulators
        const int ch = 64 * side + 32 * half + (small ? 16 * piece : 0);
        const int64_t at = (int64_t)(m[256] + tok) * p.n + m[258] * 128 + ch;
        float amax = 0.f;
        auto activate = [&](auto activation) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && small) break;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              acc[32 * h + i] = act_mul_fast(acc[32 * h + i] * rs, acc[32 * h + 16 + i] * rs, decltype(activation)::value);
              amax = fmaxf(amax, fabsf(acc[32 * h + i]));
            }
          }
        };
        if (p.activation == FMOE_ACT_GELU) activate(std::integral_constant<int, FMOE_ACT_GELU>{});
        else activate(std::integral_constant<int, FMOE_ACT_SILU>{});
        if (p.out_dtype == FMOE_E4M3) {
          // the tile's 128 channels are one quantisation group, held by four warps (M = 128: by eight)
          const int part = (small ? 4 * side : 0) + 2 * half + piece;
          float* am = amax_buf + (small ? 1024 + (small_tiles & 1) * 512 : ((ltile - small_tiles) & 1) * 512) + tok;
          const int pitch = small ? 64 : 128;
          uint64_t* bar = small ? &small_bar[warp & 1] : &amax_bar[warp & 3];
          am[part * pitch] = amax;
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar);
          if (!warp_wait(bar, (small ? small_tiles : ltile - small_tiles) & 1)) {
            report(0x7c0);
            break;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < 4 || small) amax = fmaxf(amax, am[j * pitch]);
          small_tiles += small;
          if (mine && slot >= 0) {
            const float s = group_scale(amax), r = __frcp_rn(s);
            uint32_t w[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = acc[32 * (u >> 1) + 8 * (u & 1) + i];
              const uint2 q = quant8(v, s, r, amax <= 3.0e38f);
              w[2 * u] = q.x;
              w[2 * u + 1] = q.y;
            }
            uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + at;
            if (small) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
            else store_32_bytes(dst, w, p.stores_of_32);
            if (part == 0) p.out_scale[at >> 7] = s;  // n is a multiple of 128
          }
        } else if (mine && slot >= 0) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && small) break;
            if (p.out_dtype == FMOE_F32) {
              float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at + 16 * h);
#pragma unroll
              for (int v = 0; v < 4; ++v)
                dst[v] = make_float4(acc[32 * h + 4 * v], acc[32 * h + 4 * v + 1], acc[32 * h + 4 * v + 2], acc[32 * h + 4 * v + 3]);
            } else {
              store16(reinterpret_cast<__nv_bfloat16*>(p.out) + at + 16 * h, &acc[32 * h], 1.0f, p.stores_of_32);
            }
          }
        }
      } else if (mine && slot >= 0) {
        __nv_bfloat16* obase = p.out_rows ? reinterpret_cast<__nv_bfloat16*>(p.out_rows[slot])
                                          : reinterpret_cast<__nv_bfloat16*>(p.out) + (int64_t)slot * p.n;
        const int64_t colg = (int64_t)m[258] * 256 + 128 * side + 64 * half + (small ? 32 * piece : 0);
        if (obase && colg < p.n) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= 2 && small) break;
            store16(obase + colg + 16 * c, &acc[16 * c], rs, p.stores_of_32);
          }
        }
      }
      if (PROF) prof_epi += clock64() - te0;
    }
    if (p.out_rows) __threadfence_system();  // rows stored to a peer are complete before the kernel ends
    if (PROF && threadIdx.x == 0 && blockIdx.x < 256) {
      long long* out = g_wait_prof_fp8 + (GATED ? 2048 : 0) + blockIdx.x * 8;
      out[0] = ltile;
      out[1] = prof_fw;
      out[2] = prof_fb;
      out[3] = prof_sw;
      out[4] = prof_epi;
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == kFoldWarps + 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  if (PROF && threadIdx.x == 0 && blockIdx.x < 256)
    g_wait_prof_fp8[(GATED ? 2048 : 0) + blockIdx.x * 8 + 5] = clock64() - t_kernel0;
}

template <bool GATED, bool WIDE, bool PROF, bool VEC>
int launch(const GemmParams& g, int min_rows, int max_rows, cudaStream_t st) {
  constexpr int TILE = WIDE ? 256 : TOK;
  auto kernel = WIDE ? grouped_gemm_pair_fold_wide_kernel<GATED, PROF, true, VEC> : grouped_gemm_pair_fold_kernel<GATED, PROF, true>;
  auto plain = WIDE ? grouped_gemm_pair_fold_wide_kernel<GATED, PROF, false, VEC> : grouped_gemm_pair_fold_kernel<GATED, PROF, false>;
  // setmaxnreg waits for good when the launch has fewer registers than the warps' shares add up to.  The compiler gives these
  // kernels the 96 per thread that 640 threads leave; one that gives fewer gets the kernels without the move
  // (DeepSeek-V3, 4096 tokens: 3.33 ms per layer with it, 3.40 without).
  static std::atomic<int> moves{-1};
  if (moves < 0) {
    cudaFuncAttributes fa;
    FMOE_CUDA_OK(cudaFuncGetAttributes(&fa, kernel));
    const char* env = getenv("FMOE_FOLD_MOVE_REGISTERS");  // "0": as with such a compiler
    moves = fa.numRegs * kThreads >= (kFoldWarps * kFoldRegs + 4 * kOtherRegs) * 32 && !(env && env[0] == '0');
  }
  if (!moves) kernel = plain;
  static PerDeviceOnce once_attr;  // the opt-in to > 48 KB of dynamic shared memory is per device
  const cudaError_t attr_err = per_device_once(once_attr, [&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  });
  if (attr_err != cudaSuccess)
    return fail(FMOE_ERR_CUDA, "set-up of the e4m3 kernel (smem=%d) failed: %s", kMaxSmem, cudaGetErrorString(attr_err));
  const int64_t w_rows = GATED ? 2 * g.n : g.n;
  CUtensorMap map_t, map_w;
  int rc = pair_map_tokens(&map_t, g.a, g.a_rows, g.k, 1, BOX_TOKENS);
  if (rc) return rc;
  rc = pair_map_weights(&map_w, g.w, g.num_experts, g.n, g.k, 1, GATED);
  if (rc) return rc;
  FoldParams p;
  p.sorted_token_ids = g.sorted_token_ids;
  p.expert_ids = g.expert_ids;
  p.num_tokens_post_padded = g.num_tokens_post_padded;
  p.expert_table = g.expert_table;
  p.early = g.expert_table && g.behind_late_trigger;
  p.row_scale = g.row_scale;
  p.a_scale = g.a_scale;
  p.w_scale = g.w_scale;
  p.out = g.out;
  p.out_rows = GATED ? nullptr : g.out_rows;
  p.numel = g.numel;
  p.n = g.n;
  p.w_rows = w_rows;
  p.a_scale_gather = g.a_scale_gather;
  p.top_k = g.top_k;
  p.num_experts = g.num_experts;
  p.kblocks = (int)(g.k / 128);
  p.w_tiles = (int)ceil_div<int64_t>(g.n, GATED ? 128 : 256);
  p.max_blocks = (int)g.max_blocks;
  p.activation = g.activation;
  p.group = pick_group_m(TILE, g.k);
  p.zero_padding = !g.skip_padding;
  p.out_dtype = g.out_dtype;
  p.out_scale = g.out_scale;
  p.by_expert = g.fold_by_expert && max_rows <= kNarrowRows;
  p.stores_of_32 = !p.out_rows && reinterpret_cast<uintptr_t>(g.out) % 32 == 0;  // n is a multiple of 128
  p.min_rows = min_rows;
  p.max_rows = max_rows;

  const int64_t max_tiles = g.max_blocks * ceil_div(128, TILE) * p.w_tiles;
  const int sms = device_sm_count();
  const int workers = (int)std::max<int64_t>(1, std::min<int64_t>((sms > 0 ? sms : 148) / 2, max_tiles));
  launch_pdl(kernel, dim3(2 * workers), dim3(kThreads),
             WIDE ? WideGeo::bytes(g.num_experts) : Geo<GATED>::bytes(g.num_experts), st, map_t, map_w, p);
  return launch_status("grouped_gemm_pair_fold_kernel");
}

}  // namespace

bool gemm_pair_fold_supports(const GemmParams& p, bool gated) {
  if (p.dtype != FMOE_E4M3) return false;
  if (p.out_dtype != FMOE_BF16 && !(gated && (p.out_dtype == FMOE_F32 || (p.out_dtype == FMOE_E4M3 && p.out_scale)))) return false;
  if (p.bias || p.activation == FMOE_ACT_SWIGLU_OAI) return false;  // bf16-only variant
  if (p.block_size != 128 || p.a_gather) return false;
  if (p.k <= 0 || p.k % 128 != 0 || p.n <= 0 || p.n % 128 != 0) return false;
  if (!p.a_scale || !p.w_scale) return false;
  if (!aligned16(p.a) || !aligned16(p.w) || !(aligned16(p.out) && (p.out || (!gated && p.out_rows)))) return false;
  if ((int64_t)p.num_experts * (gated ? 2 * p.n : p.n) >= (1ll << 31) || p.a_rows >= (1ll << 31)) return false;
  if (2 * p.max_blocks * ceil_div<int64_t>(p.n, gated ? 128 : 256) >= (1ll << 30) || p.num_experts > 1024) return false;
  return true;
}

int read_wait_profile_fp8(long long* host_out, int n) {
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(host_out, g_wait_prof_fp8, sizeof(long long) * (size_t)n));
  return FMOE_OK;
}

int status_word_fp8(int* out, bool clear) {
  int zero = 0;
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(out, g_device_status_fp8, sizeof(int)));
  if (clear && *out != 0) FMOE_CUDA_OK(cudaMemcpyToSymbol(g_device_status_fp8, &zero, sizeof(int)));
  return FMOE_OK;
}

int gemm_pair_fold(const GemmParams& p, bool gated, cudaStream_t st) {
  if (!gemm_pair_fold_supports(p, gated))
    return fail(FMOE_ERR_UNSUPPORTED,
                "tcgen05 fp8 gemm: needs e4m3 in, bf16 out (gate/up: or f32, or e4m3 with out_scale), block_size 128, sorted "
                "input rows, n and k multiples of 128");
  if (p.max_blocks <= 0) return FMOE_OK;
  static const bool profile = getenv("FMOE_TC_PROFILE") != nullptr;
  auto go = [&](auto wide_c, int min_rows, int max_rows) {
    constexpr bool W = decltype(wide_c)::value;
    auto with = [&](auto vec_c) {
      constexpr bool V = decltype(vec_c)::value;
      if (profile) return gated ? launch<true, W, true, V>(p, min_rows, max_rows, st) : launch<false, W, true, V>(p, min_rows, max_rows, st);
      return gated ? launch<true, W, false, V>(p, min_rows, max_rows, st) : launch<false, W, false, V>(p, min_rows, max_rows, st);
    };
    if constexpr (W) {
      if (p.k % 512 != 0 || !aligned16(p.a_scale) || !aligned16(p.w_scale)) return with(std::false_type{});
    }
    return with(std::true_type{});
  };
  constexpr int kAll = 0x7fffffff;
  // e4m3 output is the wide kernel's: a narrow tile's 128 channels are spread over both CTAs
  const bool e4m3_out = gated && p.out_dtype == FMOE_E4M3;
  if (p.fold == FoldKernel::kWide) return go(std::true_type{}, kNarrowRows + 1, kAll);
  if (e4m3_out) return go(std::true_type{}, 1, kAll);
  if (fold_narrow_only(p.numel, p.num_experts)) return go(std::false_type{}, 0, kAll);
  const int rc = go(std::false_type{}, 0, kNarrowRows);
  if (rc || p.fold == FoldKernel::kNarrow) return rc;
  return go(std::true_type{}, kNarrowRows + 1, kAll);
}

}  // namespace fmoe
