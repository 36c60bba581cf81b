// Router kernels: one warp per token.
//   fmoe_topk_softmax : softmax -> top-k -> renormalise
//   fmoe_topk_grouped : sigmoid + bias, group-limited top-k (DeepSeek-V3 style)
#include "router.cuh"

namespace fmoe {
namespace {

constexpr int kWarpsPerBlock = 4;

template <int VPT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
topk_softmax_kernel(const float* __restrict__ logits, int64_t T, int E, int k, int renorm,
                    float* __restrict__ out_w, int32_t* __restrict__ out_ids) {
  pdl_entry();
  __shared__ int s_ids[kWarpsPerBlock][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (t >= T) return;
  route_softmax<VPT>(logits + t * E, E, k, renorm, lane, s_ids[warp], out_w + t * k, out_ids + t * k);
}

// COOP (few tokens): one CTA per token; all its threads evaluate the fp64 sigmoids (one expert each instead of VPT in
// a row per lane), then warp 0 carries on alone.  Same arithmetic, shorter dependent chain.
template <int VPT, bool COOP>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
topk_grouped_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int64_t T, int E,
                    int k, int n_group, int topk_group, int renorm, float scale,
                    float* __restrict__ out_w, int32_t* __restrict__ out_ids) {
  pdl_entry();
  extern __shared__ float s_dyn[];  // per warp: score[E], choice[E]
  __shared__ int s_ids[kWarpsPerBlock][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = COOP ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  if (t >= T) return;
  float* s_score = s_dyn + (COOP ? (size_t)0 : (size_t)warp * 2 * E);
  float* s_choice = s_score + E;
  const float* row = logits + t * E;
  for (int e = COOP ? (int)threadIdx.x : lane; e < E; e += COOP ? (int)blockDim.x : 32)
    grouped_score(row[e], bias ? bias[e] : 0.f, &s_score[e], &s_choice[e]);
  if constexpr (COOP) {
    __syncthreads();
    if (warp != 0) return;
  } else {
    __syncwarp();
  }
  route_grouped<VPT>(s_score, s_choice, E, k, n_group, topk_group, renorm, scale, lane, s_ids[warp], out_w + t * k,
                     out_ids + t * k);
}

template <template <int> class Launcher, typename... Args>
int dispatch_vpt(int E, Args... args) {
  int vpt = ceil_div(E, 32);
  if (vpt <= 1) return Launcher<1>::run(args...);
  if (vpt <= 2) return Launcher<2>::run(args...);
  if (vpt <= 4) return Launcher<4>::run(args...);
  if (vpt <= 8) return Launcher<8>::run(args...);
  if (vpt <= 16) return Launcher<16>::run(args...);
  return Launcher<32>::run(args...);
}

template <int VPT>
struct SoftmaxLauncher {
  static int run(const float* logits, int64_t T, int E, int k, int renorm, float* w, int32_t* ids,
                 cudaStream_t st) {
    dim3 grid((unsigned)ceil_div<int64_t>(T, kWarpsPerBlock));
    launch_pdl(topk_softmax_kernel<VPT>, grid, dim3(kWarpsPerBlock * 32), 0, st, logits, T, E, k, renorm, w, ids);
    return launch_status("topk_softmax_kernel");
  }
};

template <int VPT>
struct GroupedLauncher {
  static int run(const float* logits, const float* bias, int64_t T, int E, int k, int n_group,
                 int topk_group, int renorm, float scale, float* w, int32_t* ids, cudaStream_t st) {
    size_t smem = (size_t)kWarpsPerBlock * 2 * E * sizeof(float);
    if (T <= 592) {  // up to four CTAs per SM: a CTA per token shortens the chain of fp64 sigmoids
                     // (E = 256: 13.3 -> 8.3 us at 1 token, 12.6 -> 8.4 us at 128 and 512)
      launch_pdl(topk_grouped_kernel<VPT, true>, dim3((unsigned)T), dim3(kWarpsPerBlock * 32), smem, st, logits, bias, T, E,
                 k, n_group, topk_group, renorm, scale, w, ids);
      return launch_status("topk_grouped_kernel");
    }
    dim3 grid((unsigned)ceil_div<int64_t>(T, kWarpsPerBlock));
    launch_pdl(topk_grouped_kernel<VPT, false>, grid, dim3(kWarpsPerBlock * 32), smem, st, logits, bias, T, E, k, n_group,
               topk_group, renorm, scale, w, ids);
    return launch_status("topk_grouped_kernel");
  }
};

}  // namespace
}  // namespace fmoe

extern "C" int fmoe_topk_softmax(const float* logits, int64_t T, int E, int k, int renormalize,
                                 float* topk_weights, int32_t* topk_ids, void* stream) {
  using namespace fmoe;
  FMOE_REQUIRE(T >= 0 && E >= 1 && E <= 1024, "topk_softmax: need 1 <= E <= 1024 (got E=%d)", E);
  FMOE_REQUIRE(k >= 1 && k <= 32 && k <= E, "topk_softmax: need 1 <= k <= min(32,E) (got k=%d, E=%d)", k, E);
  if (T == 0) return FMOE_OK;
  FMOE_REQUIRE(logits && topk_weights && topk_ids, "topk_softmax: null pointer");
  return dispatch_vpt<SoftmaxLauncher>(E, logits, T, E, k, renormalize, topk_weights, topk_ids,
                                       (cudaStream_t)stream);
}

extern "C" int fmoe_topk_grouped(const float* logits, const float* bias, int64_t T, int E, int k,
                                 int n_group, int topk_group, int renormalize, float scale,
                                 float* topk_weights, int32_t* topk_ids, void* stream) {
  using namespace fmoe;
  FMOE_REQUIRE(T >= 0 && E >= 1 && E <= 1024, "topk_grouped: need 1 <= E <= 1024 (got E=%d)", E);
  FMOE_REQUIRE(n_group >= 1 && n_group <= 32 && E % n_group == 0,
               "topk_grouped: need 1 <= n_group <= 32 dividing E (got n_group=%d, E=%d)", n_group, E);
  FMOE_REQUIRE(topk_group >= 1 && topk_group <= n_group, "topk_grouped: bad topk_group=%d", topk_group);
  FMOE_REQUIRE(k >= 1 && k <= 32 && k <= topk_group * (E / n_group),
               "topk_grouped: k=%d exceeds the experts of the kept groups", k);
  if (T == 0) return FMOE_OK;
  FMOE_REQUIRE(logits && topk_weights && topk_ids, "topk_grouped: null pointer");
  return dispatch_vpt<GroupedLauncher>(E, logits, bias, T, E, k, n_group, topk_group, renormalize, scale,
                                       topk_weights, topk_ids, (cudaStream_t)stream);
}
