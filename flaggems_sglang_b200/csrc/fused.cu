// fmoe_fused_experts: the whole expert computation behind one C call.  Host-side orchestration only:
// it carves the caller's workspace and enqueues the kernels of the other files on the given stream.
#include "align.cuh"
#include "fused.cuh"
#include "pair.cuh"
#include "rows.cuh"

#include <nvtx3/nvToolsExt.h>

namespace fmoe {

int pick_variant(int dtype, int64_t numel, int E, int64_t I, int64_t H, int forced, int* variant, int* block) {
  if (dtype == FMOE_F32) {
    if (forced != FMOE_VARIANT_AUTO && forced != FMOE_VARIANT_SIMT)
      return fail(FMOE_ERR_UNSUPPORTED, "fp32 inputs run on the simt kernels only");
    *variant = FMOE_VARIANT_SIMT;
    *block = 16;
    return FMOE_OK;
  }
  if (dtype != FMOE_BF16 && dtype != FMOE_E4M3) return fail(FMOE_ERR_INVALID_ARG, "unknown dtype %d", dtype);
  const int64_t active = std::max<int64_t>(1, std::min<int64_t>(E, numel));
  const double rows = (double)numel / (double)active;  // rows per active expert if routing were uniform
  // bf16: the tensor-core kernels cut their last column tile / zero-fill their last K step, the streaming kernel
  // masks its last 128-k chunk, so sizes such as 2880 (GPT-OSS) stay off the plain CUDA-core kernel
  const bool stream_ok = dtype == FMOE_BF16 ? (H % 16 == 0 && I % 16 == 0) : (H % 128 == 0 && I % 128 == 0);
  const bool tc_ok = dtype == FMOE_BF16 ? (I % 32 == 0 && H % 32 == 0)
                                        : (I % 128 == 0 && H % 128 == 0);
  int v = forced;
  if (v == FMOE_VARIANT_AUTO) {
    // Both families read the weights of every expert once, at about 90 % of the HBM rate, up to the rows of a streaming block:
    // from 4 to 5 rows that block doubles and the streaming kernel slows down.  Layer calls, stream / pairs in us, at 4, 5 and
    // 6 rows: Qwen3 212/207, 254/219, 262/209; half of it 117/129, 137/140, 142/132; a quarter of Mixtral 133/136, 165/136,
    // 165/136.  (The one-call layer takes the pairs at fewer rows too where they win: layer_prefers_pairs, every e4m3 call
    // among them.  The expert-parallel layer lays its receive area out by this choice.)
    if (stream_ok && ((dtype == FMOE_BF16 ? rows <= 4.0 : rows < 4.0) || !tc_ok)) v = FMOE_VARIANT_STREAM;
    else if (tc_ok) v = FMOE_VARIANT_TCGEN05;
    else v = FMOE_VARIANT_SIMT;
  }
  switch (v) {
    case FMOE_VARIANT_TCGEN05:
      if (!tc_ok) return fail(FMOE_ERR_UNSUPPORTED, "tcgen05 kernels need I %% 32 == 0 and H %% 32 == 0 (e4m3: multiples of 128)");
      *block = 128;
      break;
    case FMOE_VARIANT_STREAM:
      if (!stream_ok) return fail(FMOE_ERR_UNSUPPORTED, "stream kernels need H and I to be multiples of 16 (128 for e4m3)");
      *block = rows <= 4.0 ? 8 : (rows <= 12.0 ? 16 : 32);
      break;
    case FMOE_VARIANT_SIMT:
      *block = 16;
      break;
    default:
      return fail(FMOE_ERR_INVALID_ARG, "unknown variant %d", forced);
  }
  *variant = v;
  return FMOE_OK;
}

namespace {
inline int64_t up256(int64_t v) { return (v + 255) & ~int64_t(255); }

}

// The whole layer on the CTA-pair GEMMs although an expert has few rows.  Both families read the weights once; the pair
// kernels stream them up to 15 % faster but cost a row copy, a launch more and a longer prologue, 3-5 us.  Measured per layer,
// stream / pairs in us:
//   e4m3        DeepSeek-V3 9 tokens 510 / 447, 64 tokens 1203 / 1031, a rank's eighth with 9 to 16 tokens 262 / 243
//   not x128    (the streaming kernel masks its loads) GPT-OSS 9 tokens 232 / 183, 64 tokens 363 / 253
//   0.3 GB and more of weights (of as many experts as there are slots), 3 rows and more per expert
//               Qwen3 48 tokens 202 / 190, half of it 116 / 110; reference shape 24 tokens 248 / 233, half of it 140 / 131, a
//               quarter 87 / 79; Mixtral 12 tokens 473 / 426, a quarter 137 / 126
//   1.2 GB and more, fewer rows: H or I of 4096 and more (the streaming kernel cuts its K loop between 8 warps): 8 experts of
//               4096 x 6144 200 / 191, x 9216 311 / 291, Mixtral 431 / 388
//   fewer rows, rows below 4096: the pairs would win from 0.3 GB on here too (Qwen3 9 tokens 106 / 100, 20 157 / 150; reference shape
//               9 tokens 182 / 169, 17 243 / 225), but tests/test_abi.py holds such layers to the streaming kernels
//   0.2 GB      128 experts of 2048 x 128, 64 tokens 58 / 63; 16 of 2048 x 1024 24 tokens 50 / 52
//   below       (launches count) 32 of 1024 x 512, 24 tokens 31 / 34; 8 of 1024 x 1024 33 / 33
bool layer_prefers_pairs(const fmoe_fused_args& a, int64_t numel) {
  if (a.dtype == FMOE_E4M3) return true;  // sizes are multiples of 128
  if (a.H % 32 || a.I % 32) return false;
  if (a.H % 128 || a.I % 128) return true;
  const int64_t active = std::min<int64_t>(a.num_experts, numel), bytes = active * 6 * a.H * a.I;
  return numel >= 3 * active ? bytes >= 300000000ll : bytes >= 1200000000ll && std::max(a.H, a.I) >= 4096;
}

int plan_fused(const fmoe_fused_args& a, const RouteArgs& route, FusedPlan* pl) {
  if (a.struct_size != sizeof(fmoe_fused_args))
    return fail(FMOE_ERR_INVALID_ARG, "fused_experts: fmoe_fused_args.struct_size is %u, this library's struct has %zu "
                "bytes (binding built against another header?)", a.struct_size, sizeof(fmoe_fused_args));
  FMOE_REQUIRE(a.num_experts >= 1 && a.num_experts <= 1024 && a.top_k >= 1, "fused_experts: bad E or top_k");
  FMOE_REQUIRE(a.T >= 0 && a.H >= 1 && a.I >= 1, "fused_experts: bad sizes T=%lld H=%lld I=%lld", (long long)a.T,
               (long long)a.H, (long long)a.I);
  FMOE_REQUIRE(a.dtype == FMOE_F32 || a.dtype == FMOE_BF16 || a.dtype == FMOE_E4M3, "fused_experts: unknown dtype %d", a.dtype);
  FMOE_REQUIRE(a.activation == FMOE_ACT_SILU || a.activation == FMOE_ACT_GELU || a.activation == FMOE_ACT_SWIGLU_OAI,
               "fused_experts: unknown activation %d", a.activation);
  if (a.b1 || a.b2 || a.activation == FMOE_ACT_SWIGLU_OAI)
    FMOE_REQUIRE(a.dtype != FMOE_E4M3,
                 "fused_experts: bias and the swiglu_oai activation are not available with e4m3 weights");
  const bool channel = a.dtype == FMOE_E4M3 && a.scale_mode == FMOE_SCALE_CHANNEL;
  if (a.dtype == FMOE_E4M3) {
    FMOE_REQUIRE(a.scale_mode == FMOE_SCALE_BLOCK128 || a.scale_mode == FMOE_SCALE_CHANNEL,
                 "fused_experts: unknown scale_mode %d", a.scale_mode);
    if (channel) {
      FMOE_REQUIRE(a.H % 32 == 0 && a.I % 32 == 0 && a.H <= 16384 && a.I <= 16384,
                   "fused_experts: per-channel e4m3 needs H and I to be multiples of 32, up to 16384");
      if (a.variant != FMOE_VARIANT_AUTO && a.variant != FMOE_VARIANT_TCGEN05)
        return fail(FMOE_ERR_UNSUPPORTED, "fused_experts: per-channel e4m3 runs on the TCGEN05 kernels only");
    } else {
      FMOE_REQUIRE(a.H % 128 == 0 && a.I % 128 == 0, "fused_experts: e4m3 needs H and I to be multiples of 128");
    }
  }
  FMOE_REQUIRE(a.w_layout == FMOE_W_K_MAJOR || a.w_layout == FMOE_W_N_MAJOR || a.w_layout == FMOE_W_INTERLEAVED,
               "fused_experts: unknown w_layout %d", a.w_layout);
  if (a.w_layout == FMOE_W_INTERLEAVED && a.dtype == FMOE_E4M3)
    return fail(FMOE_ERR_UNSUPPORTED, "fused_experts: interleaved gate and up rows (FMOE_W_INTERLEAVED) need bf16 or f32 weights");
  const bool n_major = a.w_layout == FMOE_W_N_MAJOR;
  if (n_major && (a.dtype != FMOE_BF16 || a.b1 || a.b2 || a.activation == FMOE_ACT_SWIGLU_OAI ||
                  (a.variant != FMOE_VARIANT_AUTO && a.variant != FMOE_VARIANT_TCGEN05)))
    return fail(FMOE_ERR_UNSUPPORTED, "fused_experts: [E,H,2I] / [E,I,H] weights (FMOE_W_N_MAJOR) need bf16, the TCGEN05 "
                "kernels, no bias and no swiglu_oai");
  FusedPlan& p = *pl;
  p.numel = a.T * a.top_k;
  int rc = FMOE_OK;
  if (channel) {  // one kernel family: bf16-style tcgen05 pipeline on e4m3 operands, 128-row blocks
    p.variant = FMOE_VARIANT_TCGEN05;
    p.block = 128;
  } else {
    rc = pick_variant(a.dtype, p.numel, a.num_experts, a.I, a.H, n_major ? FMOE_VARIANT_TCGEN05 : a.variant, &p.variant,
                      &p.block);
    if (rc == FMOE_OK && a.variant == FMOE_VARIANT_AUTO && p.variant == FMOE_VARIANT_STREAM && layer_prefers_pairs(a, p.numel)) {
      p.variant = FMOE_VARIANT_TCGEN05;
      p.block = 128;
    }
  }
  if (rc) return rc;
  p.cap = p.numel + std::min<int64_t>(a.num_experts, p.numel) * (p.block - 1);
  p.nblk = ceil_div<int64_t>(p.cap, p.block);
  p.max_blocks = std::min<int64_t>(p.cap / p.block, p.numel);
  const int64_t eb = a.dtype == FMOE_F32 ? 4 : 2;  // element size of hidden / out / z
  const bool fp8 = a.dtype == FMOE_E4M3;
  const bool tc = p.variant == FMOE_VARIANT_TCGEN05;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    int64_t o = off;
    off += up256(bytes);
    return o;
  };
  p.off_route_ids = p.off_route_weights = -1;
  p.use_decode = plan_decode(a, route, &p.decode);
  if (p.use_decode) {
    off = p.decode.total;
    if (route.slot_of) {
      p.off_route_ids = take(p.numel * 4);
      p.off_route_weights = take(p.numel * 4);
    }
    p.total = off;
    return FMOE_OK;
  }
  if (route.logits || route.slot_of) {
    p.off_route_ids = take(p.numel * 4);
    p.off_route_weights = take(p.numel * 4);
  }
  p.off_sorted = take(p.cap * 4);
  p.off_expert = take(p.nblk * 4);
  p.off_npp = take(16);
  p.align_ws_bytes = fmoe_moe_align_workspace_bytes(p.numel, a.num_experts);
  p.off_align_ws = take(p.align_ws_bytes);
  // the CTA-pair GEMMs read the experts' rows from one table, and their tail split counts arrivals in words that the
  // align kernel clears: both GEMMs of a call have their own, so no memset stands between the kernels
  p.off_table = tc ? take(pair_table_bytes(a.num_experts)) : -1;
  p.off_counters = tc ? take(2 * kSplitCounters * 4) : -1;
  p.off_slot_pos = tc ? take(p.numel * 4) : -1;
  p.off_xs = p.off_xs_scale = p.off_actq = p.off_actq_scale = p.off_split = -1;
  p.split_bytes = 0;
  if (channel) {
    // token rows quantised straight into the sorted order, one scale per token; every row of the activation with its own
    p.off_xs = take(p.cap * a.H);
    p.off_xs_scale = take(a.T * 4);
    p.off_act = take(p.cap * a.I * 2);
    p.off_actq = take(p.cap * a.I);
    p.off_actq_scale = take(p.cap * 4);
    p.split_bytes = fmoe_gemm_split_workspace_bytes();
    p.off_split = take(p.split_bytes);
  } else if (fp8) {
    p.off_xs = take((tc ? p.cap : a.T) * a.H);
    p.off_xs_scale = take(a.T * (a.H / 128) * 4);
    // fp32 rows for the quantiser.  The wide tensor-core kernel quantises its 128-channel groups itself, so with both kernels
    // at work only experts of at most kNarrowRows rows have any (DeepSeek-V3, 16384 tokens: 134 MB, a row per position 1.34 GB)
    const bool both = tc && !fold_narrow_only(p.numel, a.num_experts);
    p.off_act = take((both ? (int64_t)a.num_experts * kNarrowRows : p.cap) * a.I * 4);
    p.off_actq = take(p.cap * a.I);
    p.off_actq_scale = take(p.cap * (a.I / 128) * 4);
  } else {
    if (tc) p.off_xs = take(p.cap * a.H * eb);
    if (tc && a.dtype == FMOE_BF16) {
      p.split_bytes = fmoe_gemm_split_workspace_bytes();
      p.off_split = take(p.split_bytes);
    }
    p.off_act = take(p.cap * a.I * eb);
  }
  p.off_z = a.no_combine ? -1 : take(p.numel * a.H * eb);
  p.total = off;
  return FMOE_OK;
}

namespace {
// Optional per-stage timing (fmoe_debug_stage_events): events of the calling thread's NEXT fused call.
thread_local void* const* t_stage_events = nullptr;
thread_local int t_stage_count = 0;

// NVTX range per stage of the layer (header-only NVTX 3: a no-op branch unless a profiler is attached).  The range that
// is open when the function returns, on an error too, is closed by the destructor.
struct StageRange {
  bool open = false;
  void next(const char* name) {
    if (open) nvtxRangePop();
    nvtxRangePushA(name);
    open = true;
  }
  ~StageRange() {
    if (open) nvtxRangePop();
  }
};
const char* const kStageNames[7] = {"fmoe.align",       "fmoe.gather_quant", "fmoe.gemm1_act", "fmoe.act_quant",
                                    "fmoe.gemm2",       "fmoe.moe_sum",      "fmoe.done"};
}  // namespace

int run_fused(const fmoe_fused_args& args, const RouteArgs& route, const FusedPlan& p, uint8_t* ws, void* stream) {
  fmoe_fused_args a = args;
  void* const* stage_ev = t_stage_events;
  const int stage_n = t_stage_count;
  t_stage_events = nullptr;
  t_stage_count = 0;
  StageRange range;
  auto mark = [&](int i) {
    if (stage_ev && i < stage_n && stage_ev[i]) cudaEventRecord((cudaEvent_t)stage_ev[i], (cudaStream_t)stream);
    if (i < 6) range.next(kStageNames[i]);
  };
  if (a.T == 0) return FMOE_OK;
  auto st = (cudaStream_t)stream;
  SortedSlots slots;
  if (route.slot_of) {
    slots.slot_of = route.slot_of;
    slots.hist = route.hist;
    slots.gate = route.gate;
    slots.ids = reinterpret_cast<int32_t*>(ws + p.off_route_ids);
    slots.weights = reinterpret_cast<float*>(ws + p.off_route_weights);
    a.topk_ids = slots.ids;
    a.topk_weights = slots.weights;
  }
  if (p.use_decode) {
    mark(0);
    if (route.slot_of) {
      AlignArgs al;
      al.numel = p.numel;
      al.E = a.num_experts;
      al.block = 1;
      const int rc = run_align_sorted(al, slots, st);
      if (rc) return rc;
    }
    const int rc = run_decode(a, route, p.decode, ws, st);
    for (int i = 1; i <= 6; ++i) mark(i);
    return rc;
  }
  if (route.logits) {
    int32_t* ids = reinterpret_cast<int32_t*>(ws + p.off_route_ids);
    float* weights = reinterpret_cast<float*>(ws + p.off_route_weights);
    const int rc = route.grouped ? fmoe_topk_grouped(route.logits, route.bias, a.T, a.num_experts, a.top_k, route.n_group,
                                                     route.topk_group, route.renorm, 1.0f, weights, ids, stream)
                                 : fmoe_topk_softmax(route.logits, a.T, a.num_experts, a.top_k, route.renorm, weights, ids, stream);
    if (rc) return rc;
    a.topk_ids = ids;
    a.topk_weights = weights;
  }
  FMOE_REQUIRE(a.hidden && a.w1 && a.w2 && a.topk_weights && a.topk_ids && (a.out || a.out_rows), "fused_experts: null pointer");
  if (a.out_rows) {
    FMOE_REQUIRE(a.no_combine && !a.zero_dropped, "fused_experts: out_rows needs no_combine = 1 and zero_dropped = 0");
    if (p.variant != FMOE_VARIANT_STREAM && p.variant != FMOE_VARIANT_TCGEN05)
      return fail(FMOE_ERR_UNSUPPORTED, "fused_experts: out_rows is taken by the STREAM and TCGEN05 kernels only");
  }
  const bool fp8 = a.dtype == FMOE_E4M3;
  const bool tc = p.variant == FMOE_VARIANT_TCGEN05;
  if (fp8) FMOE_REQUIRE(a.w1_scale && a.w2_scale, "fused_experts: e4m3 needs w1_scale and w2_scale");
  const int io = fp8 ? FMOE_BF16 : a.dtype;  // dtype of hidden / z / out
  const int64_t eb = io == FMOE_F32 ? 4 : 2;
  int32_t* sorted = reinterpret_cast<int32_t*>(ws + p.off_sorted);
  int32_t* experts = reinterpret_cast<int32_t*>(ws + p.off_expert);
  int32_t* npp = reinterpret_cast<int32_t*>(ws + p.off_npp);
  void* act = ws + p.off_act;
  void* z = a.no_combine ? a.out : (void*)(ws + p.off_z);

  mark(0);
  int32_t* table = p.off_table >= 0 ? reinterpret_cast<int32_t*>(ws + p.off_table) : nullptr;
  int32_t* counters = p.off_counters >= 0 ? reinterpret_cast<int32_t*>(ws + p.off_counters) : nullptr;
  AlignArgs al;
  al.topk_ids = a.topk_ids;
  al.numel = p.numel;
  al.E = a.num_experts;
  al.block = p.block;
  al.sorted_ids = sorted;
  al.sorted_cap = p.cap;
  al.expert_ids = experts;
  al.expert_cap = p.nblk;
  al.num_post_pad = npp;
  al.workspace = ws + p.off_align_ws;
  al.workspace_bytes = p.align_ws_bytes;
  al.table = table;
  const bool fold = fp8 && a.scale_mode == FMOE_SCALE_BLOCK128;
  al.token_tile = fold ? kNarrowRows : pick_token_tile(p.numel, a.num_experts, fp8);
  al.zero_words = counters;
  al.num_zero = counters ? 2 * kSplitCounters : 0;
  int32_t* slot_pos = tc ? reinterpret_cast<int32_t*>(ws + p.off_slot_pos) : nullptr;
  al.slot_pos = slot_pos;
  al.rows_only = tc;  // the GEMMs go by the table, the row passes by slot_pos
  al.from_sorted = route.slot_of != nullptr;
  int rc = route.slot_of ? run_align_sorted(al, slots, st) : run_align(al, st);
  if (rc) return rc;
  mark(1);
  if (a.zero_dropped) FMOE_CUDA_OK(cudaMemsetAsync(z, 0, (size_t)(p.numel * a.H * eb), st));

  GemmParams g{};
  g.struct_size = (uint32_t)sizeof(fmoe_gemm_args);
  g.w_layout = a.w_layout;
  g.variant = p.variant;
  g.num_experts = a.num_experts;
  g.top_k = a.top_k;
  g.block_size = p.block;
  g.numel = p.numel;
  g.sorted_cap = p.cap;
  g.max_blocks = p.max_blocks;
  g.sorted_token_ids = sorted;
  g.expert_ids = experts;
  g.num_tokens_post_padded = npp;

  if (p.off_split >= 0) {  // both GEMMs use it in turn (stream order)
    g.split_ws = ws + p.off_split;
    g.split_ws_bytes = p.split_bytes;
  }
  g.expert_table = table;
  g.behind_late_trigger = tc;  // below, a row pass or another pair GEMM stands before each of them
  g.token_tile = al.token_tile;
  g.skip_padding = true;  // nothing below reads a padding row's values
  GemmParams g1 = g, g2 = g;
  if (a.w_layout == FMOE_W_INTERLEAVED) g2.w_layout = FMOE_W_K_MAJOR;
  g1.split_counters = counters;
  g2.split_counters = counters ? counters + kSplitCounters : nullptr;
  g1.n = a.I;
  g1.activation = a.activation;
  g1.act_alpha = a.act_alpha;
  g1.act_limit = a.act_limit;
  g1.bias = a.b1;
  g2.bias = a.b2;
  g1.k = a.H;
  g1.w = a.w1;
  g1.out = act;
  g1.row_scale = a.apply_router_weight_on_input ? a.topk_weights : nullptr;
  g2.n = a.H;
  g2.k = a.I;
  g2.w = a.w2;
  g2.out = z;
  g2.out_rows = a.out_rows;
  g2.a_gather = 0;
  g2.a_rows = p.cap;
  g2.row_scale = a.apply_router_weight_on_input ? nullptr : a.topk_weights;
  g2.out_dtype = io;

  if (!fp8) {
    g1.dtype = g1.out_dtype = g2.dtype = a.dtype;
    if (tc) {
      void* xs = ws + p.off_xs;
      rc = run_scatter_rows(a.hidden, (int)eb, a.T, a.top_k, a.H, slot_pos, xs, st);
      if (rc) return rc;
      g1.a = xs;
      g1.a_rows = p.cap;
      g1.a_gather = 0;
    } else {
      g1.a = a.hidden;
      g1.a_rows = a.T;
      g1.a_gather = 1;
    }
    g2.a = act;
  } else {
    void* xq = ws + p.off_xs;
    float* xsc = reinterpret_cast<float*>(ws + p.off_xs_scale);
    const bool channel = a.scale_mode == FMOE_SCALE_CHANNEL;
    g1.scale_mode = g2.scale_mode = a.scale_mode;
    if (tc) {
      rc = run_quant_scatter(a.hidden, a.T, a.top_k, a.H, slot_pos, channel, xq, xsc, st);
      g1.a_scale_gather = 1;  // the gate/up GEMM looks the scales up by token
    } else {
      rc = fmoe_quant_fp8_group128(a.hidden, FMOE_BF16, a.T, a.H, nullptr, 1, 0, nullptr, xq, xsc, stream);
    }
    if (rc) return rc;
    g1.dtype = g2.dtype = FMOE_E4M3;
    g1.out_dtype = channel ? FMOE_BF16 : FMOE_F32;
    g1.a = xq;
    g1.a_scale = xsc;
    g1.a_rows = tc ? p.cap : a.T;
    g1.a_gather = tc ? 0 : 1;
    g1.w_scale = a.w1_scale;
    g2.a = ws + p.off_actq;
    g2.a_scale = reinterpret_cast<float*>(ws + p.off_actq_scale);
    g2.w_scale = a.w2_scale;
  }
  const bool both_folds = fold && tc && !fold_narrow_only(p.numel, a.num_experts);
  mark(2);
  g1.fold_by_expert = both_folds;
  if (both_folds) g1.fold = FoldKernel::kNarrow;
  rc = run_gemm(g1, true, st);
  if (rc) return rc;
  if (both_folds) {
    g1.fold = FoldKernel::kWide;
    g1.out = ws + p.off_actq;
    g1.out_scale = reinterpret_cast<float*>(ws + p.off_actq_scale);
    g1.out_dtype = FMOE_E4M3;
    rc = run_gemm(g1, true, st);
    if (rc) return rc;
  }
  mark(3);
  if (fp8) {
    float* scale = reinterpret_cast<float*>(ws + p.off_actq_scale);
    if (a.scale_mode == FMOE_SCALE_CHANNEL) {
      rc = run_quant_rows(act, p.numel, a.I, slot_pos, ws + p.off_actq, scale, st);
    } else if (tc && both_folds) {
      rc = run_quant_experts(static_cast<const float*>(act), p.numel, a.I, a.num_experts, table, kNarrowRows, ws + p.off_actq, scale, st);
    } else if (tc) {
      rc = run_quant_slots(static_cast<const float*>(act), p.numel, a.I, slot_pos, ws + p.off_actq, scale, st);
    } else {
      rc = fmoe_quant_fp8_group128(act, FMOE_F32, p.cap, a.I, sorted, 0, p.numel, npp, ws + p.off_actq, scale, stream);
    }
    if (rc) return rc;
  }
  mark(4);
  rc = run_gemm(g2, false, st);
  if (rc) return rc;
  mark(5);
  if (a.no_combine) return FMOE_OK;
  rc = fmoe_moe_sum(z, io, a.T, a.top_k, a.H, a.routed_scaling_factor == 0.f ? 1.0f : a.routed_scaling_factor, a.out, stream);
  mark(6);
  return rc;
}

int plan_within(const fmoe_fused_args& a, const RouteArgs& route, int64_t limit, bool any_rows, FusedPlan* plan) {
  const int rc = plan_fused(a, route, plan);
  if (rc || plan->total <= limit || a.variant != FMOE_VARIANT_AUTO) return rc;
  RouteArgs small = route;
  small.small_scratch = true;
  FusedPlan other;
  if (plan_fused(a, small, &other) == FMOE_OK && other.use_decode && other.total <= limit) {
    *plan = other;
    return FMOE_OK;
  }
  int variant = 0, block = 0;
  if (pick_variant(a.dtype, a.T * a.top_k, a.num_experts, a.I, a.H, FMOE_VARIANT_AUTO, &variant, &block) != FMOE_OK ||
      (variant != FMOE_VARIANT_STREAM && !any_rows))
    return FMOE_OK;
  fmoe_fused_args stream = a;
  stream.variant = FMOE_VARIANT_STREAM;
  if (plan_fused(stream, route, &other) == FMOE_OK && other.total <= limit) *plan = other;
  return FMOE_OK;
}

int run_with_workspace(const fmoe_fused_args& args, const RouteArgs& route, void* stream) {
  FusedPlan p;
  int rc = plan_within(args, route, args.workspace_bytes, false, &p);
  if (rc) return rc;
  if (args.T == 0) return FMOE_OK;
  FMOE_REQUIRE(args.workspace && (reinterpret_cast<uintptr_t>(args.workspace) & 255u) == 0,
               "fused_experts: workspace must be non-null and 256-byte aligned");
  FMOE_REQUIRE(args.workspace_bytes >= p.total, "fused_experts: workspace too small (%lld < %lld bytes)",
               (long long)args.workspace_bytes, (long long)p.total);
  return run_fused(args, route, p, reinterpret_cast<uint8_t*>(args.workspace), stream);
}

}  // namespace fmoe

extern "C" int fmoe_pick_variant(int dtype, int64_t numel, int E, int64_t I, int64_t H, int forced_variant,
                                 int* variant_out, int* block_out) {
  if (!variant_out || !block_out) return fmoe::fail(FMOE_ERR_INVALID_ARG, "pick_variant: null output pointer");
  return fmoe::pick_variant(dtype, numel, E, I, H, forced_variant, variant_out, block_out);
}

extern "C" int fmoe_debug_stage_events(void* const* events, int n) {
  if (n < 0 || n > FMOE_STAGE_EVENTS || (n > 0 && !events))
    return fmoe::fail(FMOE_ERR_INVALID_ARG, "stage events: need 0 <= n <= %d and a non-null array", FMOE_STAGE_EVENTS);
  fmoe::t_stage_events = n ? events : nullptr;
  fmoe::t_stage_count = n;
  return FMOE_OK;
}

extern "C" int64_t fmoe_fused_experts_workspace_bytes(const fmoe_fused_args* args) {
  if (!args) {
    fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_experts: args is null");
    return -1;
  }
  fmoe::FusedPlan p;
  if (fmoe::plan_fused(*args, fmoe::RouteArgs{}, &p)) return -1;
  return p.total;
}

extern "C" int fmoe_fused_experts(const fmoe_fused_args* args, void* stream) {
  using namespace fmoe;
  if (!args) return fail(FMOE_ERR_INVALID_ARG, "fused_experts: args is null");
  return run_with_workspace(*args, RouteArgs{}, stream);
}

namespace {
fmoe::RouteArgs route_args(const fmoe_route_args& r) {
  fmoe::RouteArgs out;
  out.logits = r.logits;
  out.bias = r.correction_bias;
  out.grouped = r.grouped;
  out.renorm = r.renormalize;
  out.n_group = r.n_group;
  out.topk_group = r.topk_group;
  return out;
}
int check_route(const fmoe_fused_args& a, const fmoe_route_args& r) {
  using namespace fmoe;
  FMOE_REQUIRE(r.logits, "fused_moe: logits is null");
  FMOE_REQUIRE(a.num_experts >= 1 && a.num_experts <= 1024 && a.top_k >= 1 && a.top_k <= 32 && a.top_k <= a.num_experts,
               "fused_moe: need 1 <= k <= min(32,E), E <= 1024 (got k=%d, E=%d)", a.top_k, a.num_experts);
  if (r.grouped) {
    FMOE_REQUIRE(r.n_group >= 1 && r.n_group <= 32 && a.num_experts % r.n_group == 0,
                 "fused_moe: need 1 <= n_group <= 32 dividing E (got n_group=%d, E=%d)", r.n_group, a.num_experts);
    FMOE_REQUIRE(r.topk_group >= 1 && r.topk_group <= r.n_group, "fused_moe: bad topk_group=%d", r.topk_group);
    FMOE_REQUIRE(a.top_k <= r.topk_group * (a.num_experts / r.n_group), "fused_moe: k=%d exceeds the experts of the kept groups",
                 a.top_k);
  }
  return FMOE_OK;
}
}  // namespace

extern "C" int64_t fmoe_fused_experts_sorted_workspace_bytes(const fmoe_fused_args* args) {
  if (!args) {
    fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_experts_sorted: args is null");
    return -1;
  }
  fmoe::RouteArgs r;
  const int32_t present = 0;  // the plan asks only whether there are sorted slots
  r.slot_of = &present;
  fmoe::FusedPlan p;
  if (fmoe::plan_fused(*args, r, &p)) return -1;
  return p.total;
}

extern "C" int fmoe_fused_experts_sorted(const fmoe_fused_args* args, const int32_t* topk_indx, const int32_t* expt_hist,
                                         const float* gate_scal, void* stream) {
  if (!args) return fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_experts_sorted: args is null");
  if (!topk_indx || !expt_hist || !gate_scal) return fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_experts_sorted: null pointer");
  fmoe::RouteArgs r;
  r.slot_of = topk_indx;
  r.hist = expt_hist;
  r.gate = gate_scal;
  return fmoe::run_with_workspace(*args, r, stream);
}

extern "C" int fmoe_fused_variant(const fmoe_fused_args* args, const fmoe_route_args* route, int* variant_out, int* block_out) {
  using namespace fmoe;
  if (!args || !variant_out || !block_out) return fail(FMOE_ERR_INVALID_ARG, "fused_variant: null pointer");
  if (route) {
    const int rc = check_route(*args, *route);
    if (rc) return rc;
  }
  FusedPlan p;
  const int rc = plan_fused(*args, route ? route_args(*route) : RouteArgs{}, &p);
  if (rc) return rc;
  *variant_out = p.use_decode ? FMOE_FUSED_DECODE : p.variant;
  *block_out = p.use_decode ? 0 : p.block;
  return FMOE_OK;
}

extern "C" int64_t fmoe_fused_moe_workspace_bytes(const fmoe_fused_args* args, const fmoe_route_args* route) {
  if (!args || !route) {
    fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_moe: args or route is null");
    return -1;
  }
  fmoe::FusedPlan p;
  if (check_route(*args, *route) || fmoe::plan_fused(*args, route_args(*route), &p)) return -1;
  return p.total;
}

extern "C" int fmoe_fused_moe(const fmoe_fused_args* args, const fmoe_route_args* route, void* stream) {
  if (!args || !route) return fmoe::fail(FMOE_ERR_INVALID_ARG, "fused_moe: args or route is null");
  const int rc = check_route(*args, *route);
  if (rc) return rc;
  return fmoe::run_with_workspace(*args, route_args(*route), stream);
}
