// Decode-sized layer: up to 8 tokens, bf16 or e4m3 (128x128 block scales) weights with K contiguous, two kernels.  Gate and up rows
// of w1 may alternate (FMOE_W_INTERLEAVED): the gate/up tensor map then has other strides, the box is the same.
//
// A call of this size is the reading of the chosen experts' weights and little else: 75 MB for one token of a layer with
// 8 x (2048, 768) experts, 11.7 us at the copy rate of the card.  As five or six kernels (router, align, quantiser, two
// streaming GEMMs, sum) it took 42 us: every one-CTA kernel costs 3-5 us, and each GEMM ramps its loads up and drains them.
//
//   decode_prepare_kernel : CTA 0 routes the tokens (or takes the given ids) and lists the active experts with their slots;
//                           it clears the counters; the other CTAs quantise the hidden rows (e4m3)
//   decode_layer_kernel   : one CTA per SM: 12 compute warps, a producer warp, 8 epilogue warps.  Both GEMMs in one kernel: the
//                           weights of a CTA's share of the gate/up GEMM, then of the down GEMM, stream through ONE ring of
//                           bulk copies in shared memory that keeps filling across the dependency between the two, so HBM
//                           does not idle there.  A down unit waits for its expert's activations only (a counter per
//                           expert), and the last unit of a 16-channel slab sums the slab over the slots (moe_sum).
//
// Unit: gate/up = 8 gate rows and the 8 matching up rows of one expert (one m16 tile: fragment rows g and g + 8 are a gate
// and its up value), down = 16 rows.  A stage of the ring is 1 KB of each of the 16 rows; compute warp w owns ring slot w
// and takes every stage that lands there whole, so that a warp's latency (barriers, scales, dependent MMAs) is spread over
// as many stages as the ring has (eight warps splitting every stage cost 1.1 us per 32 KB where HBM needs 0.7).  (One
// warp per slot is also what keeps the barriers' parities unambiguous: a warp free to take any stage could wait for a
// slot's round r + 1 while round r has not arrived, and pass.)  The stages' partial sums go through a
// ring in shared memory to the epilogue warps, which take the units in turn and add them in stage order: their fence and
// counter round trip last longer than a unit's stages and would hold the compute warps up.  A stage is brought by one TMA
// box of 16 KB.  The tokens' rows (later the expert's activations) stay in shared memory beside the ring.
//
// The CTAs of decode_layer_kernel wait on one another's counters, and nothing says that all of them are resident: another
// stream's kernels may hold SMs.  So the work is cut into one share per CTA and GEMM, and a CTA takes its shares from a
// counter, all gate/up shares before the first down share.  Only down shares wait, and whoever waits holds a ticket above
// every gate/up share, so that all of those belong to CTAs that run; a CTA that starts late finds less left to take.  (The
// ticket is asked for together with the block list, whose latency hides it.  One token, fixed shares / tickets: Qwen3 27.5 /
// 27.2 us per call, DeepSeek-V3 77.9 / 78.7.)  Every wait is bounded; on expiry the status word is set and the CTA finishes
// without the result.
#include "decode.cuh"
#include "fused.cuh"
#include "pair.cuh"
#include "router.cuh"
#include "rows.cuh"

namespace fmoe {

__device__ int g_device_status_decode = 0;

namespace {

constexpr int kWarps = 12;                   // compute warps: all load token rows, the first `stages` multiply
constexpr int kEpiWarps = 8;
constexpr int kThreads = (kWarps + 1 + kEpiWarps) * 32;
constexpr int ROW_BYTES = 1024;              // bytes of a weight row per stage
constexpr int PIECES = ROW_BYTES / 128;
constexpr int STAGE_BYTES = 16 * ROW_BYTES;  // [8 pieces of 128 bytes along K][16 rows], 128-byte swizzle
constexpr int MAX_STAGES = kWarps;
constexpr int kMaxRed = 160;                        // partial sums in flight (16 rows x 2, 4 or 8 tokens each)
constexpr int HEAD_BYTES = 4096;                    // barriers, flags, tickets; then the partial sums
constexpr int kMaxShares = 160;                     // shares of a GEMM, at most: one per CTA
constexpr int kHeadWords = 4 + 2 * kMaxShares + 1;  // flag, the compute warps' ticket (two in turn), all tickets a CTA can hold
static_assert((2 * kWarps + 2 * kMaxRed) * 8 + kHeadWords * 4 <= HEAD_BYTES, "shared memory");
constexpr int kMaxSmem = 227 * 1024;
constexpr int kMaxBlocks = 256;              // blocks <= slots = T * k <= 8 * 32
constexpr int x_pitch(int64_t row_bytes) { return (int)((row_bytes + 127) / 128 * 128 + 64); }

__device__ __forceinline__ void report(int code) { atomicCAS(&g_device_status_decode, 0, code); }

// plan words: [0] blocks, then per block b: expert, rows, slots[8]
__host__ __device__ constexpr int plan_expert(int b) { return 4 + b; }
__host__ __device__ constexpr int plan_rows(int b) { return 4 + kMaxBlocks + b; }
__host__ __device__ constexpr int plan_slot(int b, int i) { return 4 + 2 * kMaxBlocks + b * 8 + i; }
constexpr int kPlanWords = 4 + 10 * kMaxBlocks;

// ---------------------------------------------------------------------------------------------- prepare
struct PrepareParams {
  const float* logits;
  const float* bias;
  int grouped, renorm, n_group, topk_group;
  const int32_t* ids_in;      // given ids (logits == NULL)
  int32_t* ids;               // routed ids / weights
  float* weights;
  int32_t* plan;
  int32_t* counters;
  int num_counters;
  int T, k, E;
  const __nv_bfloat16* hidden;  // e4m3: rows to quantise
  uint8_t* xq;
  float* xs;
  int64_t H;
};

constexpr int kPrepThreads = 256;  // one per slot, of which there are at most kMaxBlocks; 8 warps route 8 tokens
static_assert(kPrepThreads >= kMaxBlocks, "one thread per slot");

template <int VPT>
__global__ void __launch_bounds__(kPrepThreads)
decode_prepare_kernel(const PrepareParams p) {
  pdl_entry();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (blockIdx.x > 0) {
    // one 128-channel group per 16-lane team
    const int groups = (int)(p.H / 128);
    const int item = (blockIdx.x - 1) * (kPrepThreads / 16) + (tid >> 4), sub = tid & 15;
    if (item >= p.T * groups) return;
    const int64_t at = (int64_t)(item / groups) * p.H + (int64_t)(item % groups) * 128 + sub * 8;
    const uint4 raw = *reinterpret_cast<const uint4*>(p.hidden + at);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    float v[8], amax = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __low2float(h[i]);
      v[2 * i + 1] = __high2float(h[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    const unsigned hmask = (tid & 16) ? 0xffff0000u : 0x0000ffffu;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(hmask, amax, off));
    const float s = group_scale(amax);
    *reinterpret_cast<uint2*>(p.xq + at) = quant8(v, s, __frcp_rn(s), amax <= 3.0e38f);
    if (sub == 0) p.xs[item] = s;
    return;
  }
  extern __shared__ float s_dyn[];  // grouped: per token score[E], choice[E]
  __shared__ int s_sel[kDecodeTokens][32];
  __shared__ int s_ids[kMaxBlocks], s_quot[kMaxBlocks], s_rem[kMaxBlocks];
  const int numel = p.T * p.k;
  for (int i = tid; i < p.num_counters; i += kPrepThreads) p.counters[i] = 0;
  if (p.logits) {
    if (p.grouped) {
      for (int i = tid; i < p.T * p.E; i += kPrepThreads) {
        const int t = i / p.E, e = i % p.E;
        grouped_score(p.logits[i], p.bias ? p.bias[e] : 0.f, &s_dyn[t * 2 * p.E + e], &s_dyn[t * 2 * p.E + p.E + e]);
      }
      __syncthreads();
    }
    if constexpr (VPT > 0) {
      if (warp < p.T) {
        if (p.grouped)
          route_grouped<VPT>(s_dyn + warp * 2 * p.E, s_dyn + warp * 2 * p.E + p.E, p.E, p.k, p.n_group, p.topk_group, p.renorm,
                             1.0f, lane, s_sel[warp], p.weights + warp * p.k, p.ids + warp * p.k);
        else
          route_softmax<VPT>(p.logits + (int64_t)warp * p.E, p.E, p.k, p.renorm, lane, s_sel[warp], p.weights + warp * p.k,
                             p.ids + warp * p.k);
        if (lane < p.k) s_ids[warp * p.k + lane] = min(max(s_sel[warp][lane], 0), p.E - 1);
      }
    }
  } else {
    for (int i = tid; i < numel; i += kPrepThreads) s_ids[i] = p.ids_in[i];
  }
  __syncthreads();
  // Blocks of at most T rows of one expert, experts ascending (one block per active expert, unless the caller's ids name
  // an expert twice for a token).  A thread per slot counts: its place among its expert's slots, then the blocks before its own.
  // (Counting by expert and a prefix sum over all of them is a chain of 8 x 5 shuffles for 256.)
  int e = -1, quot = 0, rem = -1;  // block of the expert, row in it
  if (tid < numel) {
    e = s_ids[tid];
    int before = 0;
    for (int j = 0; j < tid; ++j) before += s_ids[j] == e;
    if (e >= 0 && e < p.E) {
      quot = before / p.T;
      rem = before - quot * p.T;
    }
    s_quot[tid] = quot;
    s_rem[tid] = rem;
  }
  const int blocks = __syncthreads_count(rem == 0);
  if (tid == 0) p.plan[0] = blocks;
  if (rem >= 0) {
    int block = 0, rows = 0;
    for (int j = 0; j < numel; ++j) {
      const int ej = s_ids[j], qj = s_quot[j], rj = s_rem[j];
      block += rj == 0 && (ej < e || (ej == e && qj < quot));
      rows += rj >= 0 && ej == e && qj == quot;
    }
    p.plan[plan_slot(block, rem)] = tid;
    if (rem == 0) {
      p.plan[plan_expert(block)] = e;
      p.plan[plan_rows(block)] = rows;
    }
  }
}

// ---------------------------------------------------------------------------------------------- layer
struct LayerParams {
  const float* w1s;
  const float* w2s;
  const float* b1;
  const float* b2;
  const uint8_t* x;        // [T, H]: bf16, or e4m3
  const float* xs;         // e4m3: [T, H/128]
  const float* topk_w;     // [numel]
  const int32_t* ids;      // [numel]
  const int32_t* plan;
  void* act;               // [blocks * 8, I]: bf16, or f32 for e4m3
  __nv_bfloat16* z;        // [numel, H]
  __nv_bfloat16* out;      // [T, H]
  int32_t* ready;          // per block: gate/up units done
  int32_t* done;           // per 16-channel slab: down units done
  int32_t* tickets;        // next share: gate/up [0, shares), down [shares, 2 shares)
  int64_t H, I;
  int T, k, E, shares;
  int on_input, activation, no_combine, interleaved;
  float act_alpha, act_limit, scale;
  int stages, x_bytes;
  int n_red, n_epi, tp, red_bytes;  // partial sums in the ring, epilogue warps at work, token columns of a partial sum
};

// One 64-byte step of both operands: two MMAs, into accumulators of their own (independent chains).
__device__ __forceinline__ void mma_bf16(float (&d)[4], float (&d2)[4], const uint4& a0, const uint4& a1, const uint4& b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b.x), "r"(b.y));
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d2[0]), "+f"(d2[1]), "+f"(d2[2]), "+f"(d2[3])
      : "r"(a0.z), "r"(a1.z), "r"(a0.w), "r"(a1.w), "r"(b.z), "r"(b.w));
}
__device__ __forceinline__ void mma_e4m3(float (&d)[4], const uint4& a0, const uint4& a1, const uint4& b) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b.x), "r"(b.y));
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0.z), "r"(a1.z), "r"(a0.w), "r"(a1.w), "r"(b.z), "r"(b.w));
}
// Tiled TMA loads of one stage into this CTA's shared memory (4-D: down rows; 5-D: gate and up rows)
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(ptx::smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(ptx::smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ int32_t ld_acquire(const int32_t* p) {
  int32_t v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void compute_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory"); }  // the compute warps

// EB: bytes per weight element (2 = bf16, 1 = e4m3 with 128-block scales)
template <int EB>
__global__ void __launch_bounds__(kThreads, 1)
decode_layer_kernel(const __grid_constant__ CUtensorMap map1, const __grid_constant__ CUtensorMap map2, const LayerParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + MAX_STAGES;
  uint64_t* red_full = empty_bar + MAX_STAGES;    // [n_red] compute warp -> epilogue warp
  uint64_t* red_empty = red_full + kMaxRed;       // [n_red] epilogue warp -> compute warp
  volatile int32_t* flag = reinterpret_cast<int32_t*>(red_empty + kMaxRed);  // [0] a wait for activations gave up
  volatile int32_t* seen = flag + 2;     // [2] the compute warps' ticket, in turn
  volatile int32_t* tickets = flag + 4;  // this CTA's tickets, -1: not taken yet
  float* red = reinterpret_cast<float*>(smem + HEAD_BYTES);
  uint8_t* x_smem = smem + HEAD_BYTES + p.red_bytes;
  const uint32_t x_addr = ptx::smem_u32(x_smem);
  const uint32_t ring = x_addr + p.x_bytes;

  const int warp = ptx::uniform_warp_id(), lane = threadIdx.x & 31;
  const int stages = p.stages;
  const uint32_t n_red = p.n_red;
  if (warp == kWarps && lane == 0) {
    ptx::prefetch_tensormap(&map1);
    ptx::prefetch_tensormap(&map2);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int e = 0; e < p.n_red; ++e) {
      ptx::mbar_init(&red_full[e], 1);
      ptx::mbar_init(&red_empty[e], 1);
    }
    flag[0] = 0;
    ptx::fence_barrier_init();
  }
  for (int i = threadIdx.x; i <= 2 * kMaxShares; i += kThreads) tickets[i] = -1;
  __syncthreads();
  pdl_entry();
  int ticket0 = 0;
  if (warp == kWarps && lane == 0) ticket0 = atomicAdd(p.tickets, 1);
  const int blocks = p.plan[0];
  // Units of a share.  Gate/up: every shares-th one, so that all CTAs work on one expert after the other and at the end
  // only the last expert's activations are still to come.  Down: a contiguous piece, so that a CTA sees few experts.
  const int units1 = (int)(p.I / 8), units2 = (int)(p.H / 16), shares = p.shares;
  const int pieces1 = (int)(p.H * EB / 128), pieces2 = (int)(p.I * EB / 128);
  const int nst1 = (pieces1 + PIECES - 1) / PIECES, nst2 = (pieces2 + PIECES - 1) / PIECES;  // stages per unit
  struct Share {
    int gemm, first, step, count;
    __device__ __forceinline__ int unit(int i) const { return first + i * step; }
  };
  auto share_of = [&](int ticket) {
    // at most 256 blocks, and a token's row fits shared memory: units * shares stays far below 2^31
    const int total1 = blocks * units1, total2 = blocks * units2;
    Share s;
    s.gemm = ticket >= shares;
    const int v = ticket - s.gemm * shares;
    s.first = s.gemm ? total2 * v / shares : v;
    s.step = s.gemm ? 1 : shares;
    s.count = s.gemm ? total2 * (v + 1) / shares - s.first : (v < total1 ? (total1 - v + shares - 1) / shares : 0);
    return s;
  };
  // The CTA's idx-th ticket; 2 * shares or more: it has no further share.  Bounded like every wait.
  auto wait_ticket = [&](int idx) {
    const long long t0 = clock64();
    int t;
    while ((t = tickets[idx]) < 0) {
      if (clock64() - t0 > ptx::kWaitCycles) {
        report(0xC44);
        return 2 * shares;
      }
    }
    return t;
  };

  if (warp == kWarps) {
    // ---------------- producer: weight rows of the CTA's shares ----------------
    ticket0 = __shfl_sync(0xffffffffu, ticket0, 0);
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      int ticket = ticket0;
#pragma unroll 1
      for (int idx = 0;; ++idx) {
        if (!alive) ticket = 2 * shares;
        tickets[idx] = ticket;
        if (ticket >= 2 * shares) break;
        const Share sh = share_of(ticket);
        const int units = sh.gemm ? units2 : units1, pieces = sh.gemm ? pieces2 : pieces1;
        int next = -1;
        for (int i = 0; i < sh.count && alive; ++i) {
          // not earlier, or a CTA would take a gate/up share from one that is just starting
          if (i == sh.count - 1) next = atomicAdd(p.tickets, 1);
          const int u = sh.unit(i);
          const int e = p.plan[plan_expert(u / units)], s = u % units;
          for (int piece = 0; piece < pieces; piece += PIECES) {  // pieces past the row's end arrive as zeros
            if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
              report(0xC00 | stage);
              alive = false;
              break;
            }
            ptx::mbar_arrive_expect_tx(&full_bar[stage], STAGE_BYTES);
            if (sh.gemm == 0)
              tma_load_5d(ring + stage * STAGE_BYTES, &map1, 0, 0, p.interleaved ? 0 : 2 * e, p.interleaved ? e * units1 + s : s, piece,
                          &full_bar[stage]);
            else tma_load_4d(ring + stage * STAGE_BYTES, &map2, 0, 0, e * units2 + s, piece, &full_bar[stage]);
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
        if (sh.count == 0) next = atomicAdd(p.tickets, 1);
        ticket = next;
      }
      if (alive) {  // our own bulk copies have landed and been read before the CTA may end
        for (int s = 0; s < stages; ++s) {
          if (!ptx::mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report(0xC80 | stage);
            break;
          }
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    return;
  }

  if (warp > kWarps) {
    // ---------------- epilogue warps: units me, me + n_epi, ... of this CTA ----------------
    const int me = warp - kWarps - 1;
    bool ok = true;
    if (blocks == 0 && !p.no_combine)  // no slot has an expert: the sums are empty
      for (int64_t i = (int64_t)blockIdx.x * (kEpiWarps * 32) + me * 32 + lane; i < p.T * p.H; i += (int64_t)gridDim.x * (kEpiWarps * 32))
        p.out[i] = __float2bfloat16_rn(0.f);
    if (me >= p.n_epi) return;
    int turn = me;        // units of this CTA until this warp's next one
    uint32_t q_base = 0;  // stages before the share
#pragma unroll 1
    for (int idx = 0; ok; ++idx) {
      const int ticket = __shfl_sync(0xffffffffu, wait_ticket(idx), 0);
      if (ticket >= 2 * shares) break;
      const Share sh = share_of(ticket);
      const int gemm = sh.gemm, units = gemm ? units2 : units1, nst = gemm ? nst2 : nst1;
#pragma unroll 1
      for (; turn < sh.count && ok; turn += p.n_epi) {
        const int u = sh.unit(turn), block = u / units, s = u % units;
        const int expert = p.plan[plan_expert(block)], rows = p.plan[plan_rows(block)];
        // what the outputs need besides the sums, fetched while the stages are still landing: this lane's outputs are
        // o = lane + 32 i of [8 channels | 16 rows][tp tokens]
        const int outs = (gemm ? 16 : 8) * p.tp, tok_i = lane & (p.tp - 1), row_i = lane / p.tp, row_step = 32 / p.tp;
        const int32_t slot = tok_i < rows ? p.plan[plan_slot(block, tok_i)] : -1;
        const float wt = (slot >= 0 && p.on_input == !gemm) ? p.topk_w[slot] : 1.0f;
        // the unit's partial sums, in stage order
        const uint32_t q0 = q_base + (uint32_t)(turn * nst);
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, sum_up[2] = {0.f, 0.f};
        for (int st = 0; st < nst; ++st) {
          const uint32_t q = q0 + st;
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&red_full[q % n_red], (q / n_red) & 1));
          if (!ok) {
            report(0xC10 | me);
            break;
          }
          const float* part = red + (q % n_red) * 16 * p.tp;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (lane + 32 * i < outs) sum[i] += part[lane + 32 * i];
          if (gemm == 0) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
              if (lane + 32 * i < outs) sum_up[i] += part[8 * p.tp + lane + 32 * i];
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&red_empty[q % n_red]);
        }
        if (!ok) break;
        if (gemm == 0) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (slot >= 0 && lane + 32 * i < outs) {
              const int64_t ch = (int64_t)s * 8 + row_i + row_step * i;
              const float* bias = p.b1 ? p.b1 + (int64_t)expert * 2 * p.I + (p.interleaved ? 2 * ch : ch) : nullptr;
              const float o = gated_output<false>(sum[i], sum_up[i], bias ? bias[0] : 0.f, bias ? bias[p.interleaved ? 1 : p.I] : 0.f, wt,
                                                  p.activation, p.act_alpha, p.act_limit);
              const int64_t at = ((int64_t)block * 8 + tok_i) * p.I + ch;
              if constexpr (EB == 2) reinterpret_cast<__nv_bfloat16*>(p.act)[at] = __float2bfloat16_rn(o);
              else reinterpret_cast<float*>(p.act)[at] = o;
            }
          }
          __threadfence();  // the activations are visible device-wide before the unit counts
          __syncwarp();
          if (lane == 0) atomicAdd(p.ready + block, 1);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (slot >= 0 && lane + 32 * i < outs) {
              const int64_t ch = (int64_t)s * 16 + row_i + row_step * i;
              p.z[(int64_t)slot * p.H + ch] = __float2bfloat16_rn((sum[i] + (p.b2 ? p.b2[(int64_t)expert * p.H + ch] : 0.f)) * wt);
            }
          }
          if (p.no_combine) continue;
          __threadfence();
          __syncwarp();
          int last = 0;
          if (lane == 0) last = atomicAdd(p.done + s, 1) == blocks - 1;
          if (__shfl_sync(0xffffffffu, last, 0)) {
            // the slab's last unit: out[t] = sum over the token's slots, in slot order
            __threadfence();
            for (int i = lane; i < p.T * 16; i += 32) {
              const int tok = i >> 4;
              const int64_t ch = (int64_t)s * 16 + (i & 15);
              float a = 0.f;
#pragma unroll 8
              for (int j = 0; j < p.k; ++j) {
                const int sl = tok * p.k + j, e = p.ids[sl];
                const unsigned short v = __ldcg(reinterpret_cast<const unsigned short*>(p.z) + (int64_t)sl * p.H + ch);
                if (e >= 0 && e < p.E) a += __bfloat162float(__ushort_as_bfloat16(v));
              }
              __nv_bfloat16 o = __float2bfloat16_rn(a);
              if (p.scale != 1.0f) o = __float2bfloat16_rn(__bfloat162float(o) * p.scale);
              p.out[(int64_t)tok * p.H + ch] = o;
            }
          }
        }
      }
      turn -= sh.count;
      q_base += (uint32_t)(sh.count * nst);
    }
    return;
  }

  // ---------------- compute warps ----------------
  const int tid = threadIdx.x, g = lane >> 2, t = lane & 3;
  bool ok = true;
  uint32_t q_base = 0;  // stages before the share
#pragma unroll 1
  for (int idx = 0;; ++idx) {
    // One thread waits for the ticket, so that all compute warps act on the same one, also when it does not come
    if (tid == 0) seen[idx & 1] = wait_ticket(idx);
    compute_barrier();
    const int ticket = seen[idx & 1];
    if (ticket >= 2 * shares) break;
    const Share sh = share_of(ticket);
    const int gemm = sh.gemm, units = gemm ? units2 : units1, count = sh.count, nst = gemm ? nst2 : nst1;
    const int pieces = gemm ? pieces2 : pieces1, kblocks = (int)((gemm ? p.I : p.H) / 128);
    const uint32_t row_bytes = (uint32_t)pieces * 128;
    const int xp = x_pitch(row_bytes);
    float* x_scale = nullptr;  // e4m3: scales of the rows in shared memory, [row][kblocks]
    if constexpr (EB == 1) x_scale = reinterpret_cast<float*>(x_smem + p.T * xp);
    if (gemm == 0 && idx == 0) {  // the tokens' rows, once: all gate/up shares come before the first down share
      const int vecs = (int)(row_bytes / 16);
      for (int i = tid; i < p.T * vecs; i += kWarps * 32) {
        const int r = i / vecs, c = i % vecs;
        *reinterpret_cast<uint4*>(x_smem + r * xp + c * 16) =
            __ldg(reinterpret_cast<const uint4*>(p.x + (int64_t)r * row_bytes) + c);
      }
      if constexpr (EB == 1)
        for (int i = tid; i < p.T * kblocks; i += kWarps * 32) x_scale[i] = __ldg(p.xs + i);
      compute_barrier();
    }
    // gate/up: all units in one go; down: block by block, each with its expert's activations in shared memory
#pragma unroll 1
    for (int seg = 0; seg < count;) {
      const int seg_end = gemm ? min(count, (sh.unit(seg) / units + 1) * units - sh.first) : count;
      if (gemm == 1) {
        const int block = sh.unit(seg) / units, rows = p.plan[plan_rows(block)];
        if (tid == 0) {  // every gate/up unit of the block has been published
          const long long t0 = clock64();
          while (ld_acquire(p.ready + block) < units1) {
            if (clock64() - t0 > ptx::kWaitCycles) {
              report(0xC40);
              flag[0] = 1;
              break;
            }
          }
        }
        compute_barrier();  // also: the token rows, or the previous block's, have been read by everyone
        if (flag[0]) ok = false;
        if constexpr (EB == 2) {
          const int vecs = (int)(row_bytes / 16);
          const uint4* src = reinterpret_cast<const uint4*>(p.act) + (int64_t)block * 8 * vecs;
          for (int i = tid; i < rows * vecs; i += kWarps * 32)
            *reinterpret_cast<uint4*>(x_smem + (i / vecs) * xp + (i % vecs) * 16) = __ldcg(src + i);
        } else {
          // quantised here, 16 lanes per 128-channel group
          const float* src = reinterpret_cast<const float*>(p.act) + (int64_t)block * 8 * p.I;
          const int sub = tid & 15;
          const unsigned hmask = (tid & 16) ? 0xffff0000u : 0x0000ffffu;
          for (int i = tid >> 4; i < rows * kblocks; i += kWarps * 2) {
            const int r = i / kblocks, kb = i % kblocks;
            const float4* q = reinterpret_cast<const float4*>(src + (int64_t)r * p.I + kb * 128 + sub * 8);
            const float4 a = __ldcg(q), b = __ldcg(q + 1);
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            float amax = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(hmask, amax, off));
            const float sc = group_scale(amax);
            *reinterpret_cast<uint2*>(x_smem + r * xp + kb * 128 + sub * 8) = quant8(v, sc, __frcp_rn(sc), amax <= 3.0e38f);
            if (sub == 0) x_scale[r * kblocks + kb] = sc;
          }
        }
        compute_barrier();
      }
      int cached = -1, expert = 0, rows = 0;
      int32_t slot_g = -1, slot_t[2] = {-1, -1};
      const uint32_t first = q_base + (uint32_t)seg * nst, last = q_base + (uint32_t)seg_end * nst;
      // stage q lands in ring slot q % stages and belongs to the warp of that number
#pragma unroll 1
      for (uint32_t q = first + (warp + stages - first % stages) % stages; q < last && warp < stages; q += stages) {
        const int u = sh.unit((int)((q - q_base) / nst)), st = (int)((q - q_base) % nst), block = u / units;
        if (block != cached) {
          cached = block;
          expert = p.plan[plan_expert(block)];
          rows = p.plan[plan_rows(block)];
          slot_g = g < rows ? p.plan[plan_slot(block, g)] : -1;
#pragma unroll
          for (int j = 0; j < 2; ++j) slot_t[j] = 2 * t + j < rows ? p.plan[plan_slot(block, 2 * t + j)] : -1;
        }
        // shared-memory rows of this lane's tokens: the token's row (gate/up) or the row within the block (down)
        const bool has = slot_g >= 0;
        const uint32_t xrow = x_addr + (gemm ? g : (has ? slot_g / p.k : 0)) * xp + t * 16 + st * ROW_BYTES;
        const int n_pieces = min(PIECES, pieces - PIECES * st);
        float sw = 0.f;  // e4m3: lane 16 h + j holds the weight scale of K block j of fragment rows g (h = 0) and g + 8
        const float* sa[2] = {nullptr, nullptr};
        if constexpr (EB == 1) {
          const int s = u % units, kb = PIECES * st + (lane & 15);
          const float* row = gemm ? p.w2s + ((int64_t)expert * (p.H / 128) + s / 8) * kblocks
                                  : p.w1s + ((int64_t)expert * (2 * p.I / 128) + s / 16 + (lane >> 4) * (p.I / 128)) * kblocks;
          if ((lane & 15) < n_pieces) sw = __ldg(row + kb);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            sa[j] = x_scale + (slot_t[j] < 0 ? 0 : (gemm ? 2 * t + j : slot_t[j] / p.k)) * kblocks + PIECES * st;
        }
        const int slot = warp;
        if (ok && !__all_sync(0xffffffffu, ptx::mbar_wait(&full_bar[slot], (q / stages) & 1))) {
          report(0xC20 | slot);
          ok = false;
        }
        const uint32_t wrow = ring + slot * STAGE_BYTES + g * 128;
        float acc[4][4] = {};  // bf16: four independent chains of MMAs
#pragma unroll(EB == 2 ? 4 : 2)
        for (int pc = 0; pc < n_pieces; ++pc) {
          float part[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t w = wrow + pc * 2048 + (((i * 4 + t) ^ g) << 4);  // swizzled 16-byte unit of row g
            const uint4 a0 = lds128(w), a1 = lds128(w + 1024);
            const uint4 b = has ? lds128(xrow + pc * 128 + i * 64) : make_uint4(0, 0, 0, 0);
            if constexpr (EB == 2) mma_bf16(acc[2 * i], acc[2 * i + 1], a0, a1, b);
            else mma_e4m3(part[i], a0, a1, b);
          }
          if constexpr (EB == 1) {
            const float w0 = __shfl_sync(0xffffffffu, sw, pc), w1 = gemm ? w0 : __shfl_sync(0xffffffffu, sw, 16 + pc);
            const float a0 = slot_t[0] >= 0 ? sa[0][pc] : 0.f, a1 = slot_t[1] >= 0 ? sa[1][pc] : 0.f;
            acc[0][0] = fmaf(part[0][0] + part[1][0], a0 * w0, acc[0][0]);
            acc[0][1] = fmaf(part[0][1] + part[1][1], a1 * w0, acc[0][1]);
            acc[0][2] = fmaf(part[0][2] + part[1][2], a0 * w1, acc[0][2]);
            acc[0][3] = fmaf(part[0][3] + part[1][3], a1 * w1, acc[0][3]);
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&empty_bar[slot]);
        // partial sums to the epilogue: accumulator j of lane (g, t) is row g + 8 * (j >> 1), token 2t + (j & 1)
        const int buf = q % n_red;
        if (ok && !__all_sync(0xffffffffu, ptx::mbar_wait(&red_empty[buf], ((q / n_red) & 1) ^ 1))) {
          report(0xC18);
          ok = false;
        }
        if constexpr (EB == 2) {
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[0][j] = (acc[0][j] + acc[1][j]) + (acc[2][j] + acc[3][j]);
        }
        if (2 * t < p.tp) {
          float* mine = red + buf * 16 * p.tp + 2 * t;
          *reinterpret_cast<float2*>(mine + g * p.tp) = make_float2(acc[0][0], acc[0][1]);
          *reinterpret_cast<float2*>(mine + (g + 8) * p.tp) = make_float2(acc[0][2], acc[0][3]);
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&red_full[buf]);
      }
      seg = seg_end;
    }
    q_base += (uint32_t)(count * nst);
  }
}

thread_local int t_debug_ctas = 0;  // fmoe_debug_decode_ctas

template <int VPT>
int launch_prepare(const PrepareParams& p, int quant_ctas, size_t smem, cudaStream_t st) {
  launch_pdl(decode_prepare_kernel<VPT>, dim3(1 + quant_ctas), dim3(kPrepThreads), smem, st, p);
  return launch_status("decode_prepare_kernel");
}

template <int EB>
int launch_layer(const fmoe_fused_args& a, const LayerParams& p, int smem, cudaStream_t st) {
  static PerDeviceOnce once_attr;
  const cudaError_t err = per_device_once(once_attr, [] {
    return cudaFuncSetAttribute(decode_layer_kernel<EB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  });
  if (err != cudaSuccess) return fail(FMOE_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(err));
  // 128-byte pieces of 8 gate rows and their 8 up rows (gate and up halves of all experts in one dimension; where they
  // alternate, the groups of 16 rows of all experts) / of 16 rows
  constexpr int PIECE = 128 / EB;
  const cuuint64_t row1 = (cuuint64_t)a.H * EB, row2 = (cuuint64_t)a.I * EB;
  const cuuint64_t E = a.num_experts, groups = (cuuint64_t)a.I / 8;
  const cuuint64_t dims1[5] = {PIECE, 8, p.interleaved ? 2 : 2 * E, p.interleaved ? E * groups : groups, row1 / 128};
  const cuuint64_t strides1[4] = {p.interleaved ? row1 * 2 : row1, p.interleaved ? row1 : row1 * a.I,
                                  p.interleaved ? row1 * 16 : row1 * 8, 128};
  const cuuint32_t box1[5] = {PIECE, 8, 2, 1, PIECES};
  const cuuint64_t dims2[4] = {PIECE, 16, (cuuint64_t)a.num_experts * (a.H / 16), row2 / 128};
  const cuuint64_t strides2[3] = {row2, row2 * 16, 128};
  const cuuint32_t box2[4] = {PIECE, 16, 1, PIECES};
  CUtensorMap map1, map2;
  int rc = encode_tensor_map(&map1, a.w1, EB, 5, dims1, strides1, box1, true, "decode gate/up weights");
  if (rc) return rc;
  rc = encode_tensor_map(&map2, a.w2, EB, 4, dims2, strides2, box2, true, "decode down weights");
  if (rc) return rc;
  const int sms = device_sm_count();
  LayerParams q = p;
  q.shares = std::min(sms > 0 ? sms : 148, kMaxShares);
  const int ctas = t_debug_ctas > 0 ? std::min(t_debug_ctas, q.shares) : q.shares;
  t_debug_ctas = 0;
  launch_pdl(decode_layer_kernel<EB>, dim3(ctas), dim3(kThreads), (size_t)smem, st, map1, map2, q);
  return launch_status("decode_layer_kernel");
}

}  // namespace

int status_word_decode(int* out, bool clear) {
  int zero = 0;
  FMOE_CUDA_OK(cudaMemcpyFromSymbol(out, g_device_status_decode, sizeof(int)));
  if (clear && *out != 0) FMOE_CUDA_OK(cudaMemcpyToSymbol(g_device_status_decode, &zero, sizeof(int)));
  return FMOE_OK;
}

namespace {

// e4m3 layers of up to 8 tokens that the CTA-pair kernels run faster.  They need a list, a row copy, a quantiser and a combine pass
// more, some 15 us, and nearly the same time whatever the tokens.  The decode kernels pay for token rows: long ones leave the ring
// few stages, every token column has scale products of its own, a down row of less than ROW_BYTES fills part of a stage, and every
// active expert costs 1-3 us of waits.  With cold weights, decode / pairs in us:
//   k = 8, E = 256 (token rows decide): H = 7168, I = 1024: 3 tokens 110 / 115, 4 135 / 135, 8 263 / 226; I = 512: 2 61 / 56, 4 101 /
//               82, 8 181 / 136; I = 256: 2 53 / 46, 4 81 / 60; H = 4096, I = 1536: 4 109 / 115, 8 210 / 189
//   few slots   (launches and prologues count): H = 7168, I = 256: E = 8, k = 2, 3 tokens 30 / 36, 4 33 / 37, 5 37 / 37, 8 41 / 38; E = 16,
//               k = 1, 3 tokens 23 / 35, 8 36 / 37; I = 128: E = 8, k = 2, 5 tokens 31 / 36, 8 36 / 36; E = 32, k = 4, 3 tokens 41 / 38;
//               I = 1024: E = 16, k = 1, 5 tokens 41 / 41, 6 46 / 43; I = 1792: 8 tokens 61 / 65
//               H = 4096, I = 256: E = 8, k = 2, 8 tokens 29 / 31; E = 16, k = 2, 6 tokens 30 / 31, 8 32 / 31; E = 32, k = 4, 5 tokens 38 / 33
// Of 741 calls past the first line (H of 4096 to 7168, I of 128 to 1792, k of 1 to 8), 252 took 2 to 69 % longer on the pairs.  By
// the lines below 21 still do, 2 to 8 %, and 17 take 2 to 7 % longer on the decode kernels.
// Whole down rows (H = 7168, I = 2048) stay with the decode kernels although only 1 to 4 tokens gain by it (76 / 87, 225 / 234; 5
// tokens 305 / 271, 8 434 / 369): tests/test_abi.py holds fmoe_fused_variant to them for 8 tokens of that layer.  bf16 layers
// stay too (Qwen3 90 / 95, Mixtral 367 / 366, GPT-OSS 168 / 174 with 8 tokens).
bool pairs_are_faster(const fmoe_fused_args& a) {
  if (a.I >= 2048 || a.T * a.H <= (a.I >= 512 ? 24576 : 16384)) return false;
  // channels of the token rows and of the slots' rows; from I = 1536 on the pairs' tiles need a second round
  const int64_t rows = a.T * (a.top_k + 1) * a.H;
  if (rows <= (a.I >= 1536 ? 112 : (a.I > 512 ? 76 : 88)) * 1024) return false;
  const int64_t weights = std::min<int64_t>(a.num_experts, a.T * a.top_k) * 3 * a.H * a.I;
  return weights > 28000000 || rows > 128 * 1024;
}

}  // namespace

bool plan_decode(const fmoe_fused_args& a, const RouteArgs& r, DecodePlan* pl) {
  const bool fp8 = a.dtype == FMOE_E4M3;
  if (a.variant != FMOE_VARIANT_AUTO || (a.w_layout != FMOE_W_K_MAJOR && a.w_layout != FMOE_W_INTERLEAVED) || a.out_rows) return false;
  if (a.dtype != FMOE_BF16 && !(fp8 && a.scale_mode == FMOE_SCALE_BLOCK128)) return false;
  if (a.no_combine && a.zero_dropped) return false;
  if (a.T < 1 || a.T > kDecodeTokens || a.top_k > 32 || a.num_experts > 1024) return false;
  if (a.H % (fp8 ? 128 : 64) || a.I % (fp8 ? 128 : 64)) return false;  // rows of whole 128-byte pieces
  if (fp8 && !r.small_scratch && pairs_are_faster(a)) return false;
  if (r.logits && (a.num_experts > 256 || (r.grouped && (int64_t)a.T * a.num_experts * 8 > 32 * 1024))) return false;
  const int eb = fp8 ? 1 : 2;
  // token rows of the gate/up GEMM; rows of one block (at most T) of the down GEMM
  auto rows_bytes = [&](int64_t rows, int64_t K) {
    const int64_t b = rows * x_pitch(K * eb);
    return fp8 ? b + rows * (K / 128) * 4 : b;
  };
  const int64_t x = (std::max(rows_bytes(a.T, a.H), rows_bytes(a.T, a.I)) + 1023) / 1024 * 1024;
  // Partial sums in flight.  An epilogue warp may wait for the last stage of a unit n_epi units ahead of the oldest one
  // whose stages are still landing (at most two rounds of the ring): that span has to fit, or a parity would repeat.
  const int nst = (int)ceil_div<int64_t>(std::max(a.H, a.I) * eb, ROW_BYTES);
  // Rows of more than 9 stages get a longer ring, for four epilogue warps at work (one, with Mixtral's 28 stages per row of
  // the down projection, took 213 us for one token).
  pl->n_red = std::min(kMaxRed, std::max(64, 2 * MAX_STAGES + 4 + 4 * nst));
  pl->n_epi = std::min(kEpiWarps, (pl->n_red - 2 * MAX_STAGES - 4) / nst);
  if (pl->n_epi < 1) return false;
  pl->tp = a.T <= 2 ? 2 : (a.T <= 4 ? 4 : 8);
  pl->red_bytes = (pl->n_red * 16 * pl->tp * 4 + 1023) / 1024 * 1024;
  const int64_t left = kMaxSmem - HEAD_BYTES - pl->red_bytes - x;
  // six stages (96 KB in flight per SM) still stream near the HBM rate; with less room other kernels are the better choice
  if (left < 6 * STAGE_BYTES) return false;
  pl->stages = (int)std::min<int64_t>(left / STAGE_BYTES, MAX_STAGES);
  pl->x_bytes = (int)x;
  pl->smem = (int)(HEAD_BYTES + pl->red_bytes + x + pl->stages * STAGE_BYTES);
  const int64_t numel = a.T * a.top_k, blocks = numel;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    const int64_t o = off;
    off += (bytes + 255) & ~int64_t(255);
    return o;
  };
  pl->off_plan = take(kPlanWords * 4);
  pl->off_ids = take(numel * 4);
  pl->off_weights = take(numel * 4);
  pl->off_xq = fp8 ? take(a.T * a.H) : 0;
  pl->off_xs = fp8 ? take(a.T * (a.H / 128) * 4) : 0;
  pl->off_act = take(blocks * 8 * a.I * (fp8 ? 4 : 2));
  pl->off_z = a.no_combine ? 0 : take(numel * a.H * 2);
  pl->off_counters = take((kMaxBlocks + a.H / 16 + 1) * 4);
  pl->total = off;
  return true;
}

int run_decode(const fmoe_fused_args& a, const RouteArgs& r, const DecodePlan& pl, uint8_t* ws, cudaStream_t st) {
  const bool fp8 = a.dtype == FMOE_E4M3;
  FMOE_REQUIRE(a.hidden && a.w1 && a.w2 && a.out && (r.logits || (a.topk_weights && a.topk_ids)), "fused_experts: null pointer");
  FMOE_REQUIRE(!fp8 || (a.w1_scale && a.w2_scale), "fused_experts: e4m3 needs w1_scale and w2_scale");
  FMOE_REQUIRE(aligned16(a.hidden) && aligned16(a.w1) && aligned16(a.w2) && aligned16(a.out), "fused_experts: misaligned pointer");
  PrepareParams q{};
  q.logits = r.logits;
  q.bias = r.bias;
  q.grouped = r.grouped;
  q.renorm = r.renorm;
  q.n_group = r.n_group;
  q.topk_group = r.topk_group;
  q.ids_in = a.topk_ids;
  q.ids = reinterpret_cast<int32_t*>(ws + pl.off_ids);
  q.weights = reinterpret_cast<float*>(ws + pl.off_weights);
  q.plan = reinterpret_cast<int32_t*>(ws + pl.off_plan);
  q.counters = reinterpret_cast<int32_t*>(ws + pl.off_counters);
  q.num_counters = kMaxBlocks + (int)(a.H / 16) + 1;
  q.T = (int)a.T;
  q.k = a.top_k;
  q.E = a.num_experts;
  q.hidden = static_cast<const __nv_bfloat16*>(a.hidden);
  q.xq = ws + pl.off_xq;
  q.xs = reinterpret_cast<float*>(ws + pl.off_xs);
  q.H = a.H;
  const int quant_ctas = fp8 ? (int)ceil_div<int64_t>(a.T * (a.H / 128), kPrepThreads / 16) : 0;
  const size_t smem = (r.logits && r.grouped) ? (size_t)a.T * 2 * a.num_experts * sizeof(float) : 0;
  const int vpt = r.logits ? ceil_div(a.num_experts, 32) : 0;
  int rc = vpt == 0   ? launch_prepare<0>(q, quant_ctas, smem, st)
           : vpt <= 1 ? launch_prepare<1>(q, quant_ctas, smem, st)
           : vpt <= 2 ? launch_prepare<2>(q, quant_ctas, smem, st)
           : vpt <= 4 ? launch_prepare<4>(q, quant_ctas, smem, st)
                      : launch_prepare<8>(q, quant_ctas, smem, st);
  if (rc) return rc;
  LayerParams p{};
  p.w1s = a.w1_scale;
  p.w2s = a.w2_scale;
  p.b1 = a.b1;
  p.b2 = a.b2;
  p.x = fp8 ? q.xq : static_cast<const uint8_t*>(a.hidden);
  p.xs = q.xs;
  p.topk_w = r.logits ? q.weights : a.topk_weights;
  p.ids = r.logits ? q.ids : a.topk_ids;
  p.plan = q.plan;
  p.act = ws + pl.off_act;
  p.z = static_cast<__nv_bfloat16*>(a.no_combine ? a.out : (void*)(ws + pl.off_z));
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.ready = q.counters;
  p.done = q.counters + kMaxBlocks;
  p.tickets = p.done + a.H / 16;
  p.H = a.H;
  p.I = a.I;
  p.T = (int)a.T;
  p.k = a.top_k;
  p.E = a.num_experts;
  p.on_input = a.apply_router_weight_on_input;
  p.activation = a.activation;
  p.no_combine = a.no_combine;
  p.interleaved = a.w_layout == FMOE_W_INTERLEAVED;
  p.act_alpha = a.act_alpha;
  p.act_limit = a.act_limit;
  p.scale = a.routed_scaling_factor == 0.f ? 1.0f : a.routed_scaling_factor;
  p.stages = pl.stages;
  p.x_bytes = pl.x_bytes;
  p.n_red = pl.n_red;
  p.n_epi = pl.n_epi;
  p.tp = pl.tp;
  p.red_bytes = pl.red_bytes;
  return fp8 ? launch_layer<1>(a, p, pl.smem, st) : launch_layer<2>(a, p, pl.smem, st);
}

}  // namespace fmoe

extern "C" int fmoe_debug_decode_ctas(int ctas) {
  if (ctas < 0) return fmoe::fail(FMOE_ERR_INVALID_ARG, "decode CTAs: need 0 (no limit) or more");
  fmoe::t_debug_ctas = ctas;
  return FMOE_OK;
}
