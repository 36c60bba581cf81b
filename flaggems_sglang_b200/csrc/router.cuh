// Routing of one token by one warp, shared by the router kernels (router.cu) and the decode layer (decode.cu).
// Expert e of a token lives in lane e % 32, register e / 32 (coalesced loads).
// NaN contract: a NaN logit (or a NaN biased score) ranks as -inf, ties go to the lower index, and a softmax row
// without any logit above -inf is routed as if all its logits were equal; every id written is inside [0, E).
#pragma once
#include "common.cuh"

namespace fmoe {

#if defined(__CUDACC__)
#define kNegInf (__int_as_float(0xff800000))

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Unsigned integers in the order of the floats (-0 counts as +0; no NaN); every value is above 0.
__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t b = __float_as_uint(v + 0.0f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// Index of the largest key of the warp, ties to the lower index.  Two warp reductions in hardware (redux.sync) instead
// of ten dependent shuffles: a top-8 of 256 experts is a chain of eight of these.
__device__ __forceinline__ int warp_argmax(uint32_t key, int idx) {
  const uint32_t best = __reduce_max_sync(0xffffffffu, key);
  return (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)idx : 0x7fffffffu);
}

// k rounds of warp-wide argmax over the per-lane register file `key`; sel_ids[j] = winner of round j.
template <int VPT>
__device__ __forceinline__ void select_topk(const float (&key)[VPT], int E, int k, int lane, int* sel_ids) {
  uint32_t u[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) u[i] = (lane + 32 * i) < E ? ordered_bits(key[i]) : 0u;  // 0: cannot win again
  for (int j = 0; j < k; ++j) {
    uint32_t bu = 0;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (u[i] > bu) {  // ascending index: a tie keeps the lower one
        bu = u[i];
        bi = lane + 32 * i;
      }
    }
    const int id = warp_argmax(bu, bi);
    if (lane == 0) sel_ids[j] = id;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if (lane + 32 * i == id) u[i] = 0u;
  }
}

// softmax -> top-k -> optional renormalisation of one row of logits; s_ids: 32 ints of shared memory of this warp.
template <int VPT>
__device__ __forceinline__ void route_softmax(const float* __restrict__ row, int E, int k, int renorm, int lane, int* s_ids,
                                              float* __restrict__ out_w, int32_t* __restrict__ out_ids) {
  float key[VPT];
  float mx = kNegInf;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int e = lane + 32 * i;
    const float v = (e < E) ? row[e] : kNegInf;
    key[i] = (v != v) ? kNegInf : v;  // NaN ranks as -inf
    mx = fmaxf(mx, key[i]);
  }
  mx = warp_max(mx);
  if (mx == kNegInf) {  // no logit above -inf: equal logits (uniform probabilities, experts 0..k-1)
    mx = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if (lane + 32 * i < E) key[i] = 0.f;
  }
  float denom = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    if (lane + 32 * i < E) denom += expf(key[i] - mx);
  denom = warp_sum(denom);

  select_topk<VPT>(key, E, k, lane, s_ids);
  __syncwarp();
  // lane j owns winner j
  int id = (lane < k) ? min(max(s_ids[lane], 0), E - 1) : 0;
  // the winner's (sanitised) logit lives in lane id % 32, register id / 32
  float kv = kNegInf;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const float cand = __shfl_sync(0xffffffffu, key[i], id & 31);
    if (i == (id >> 5)) kv = cand;
  }
  float p = (lane < k) ? __fdiv_rn(expf(kv - mx), denom) : 0.f;
  if (renorm) {
    float s = 0.f;
    for (int j = 0; j < k; ++j) s += __shfl_sync(0xffffffffu, p, j);  // sequential, j ascending
    p = __fdiv_rn(p, s);
  }
  if (lane < k) {
    out_w[lane] = p;
    out_ids[lane] = id;
  }
}

// Sigmoid score of expert e and the choice value it is ranked by (correctly rounded fp32 sigmoid: fp64, rounded once).
__device__ __forceinline__ void grouped_score(float lg, float bias, float* score, float* choice) {
  double z = (lg != lg) ? -INFINITY : (double)lg;  // NaN ranks as -inf (score 0)
  float s = (float)(1.0 / (1.0 + exp(-z)));
  float c = s + bias;
  if (c != c) c = kNegInf;
  *score = s;
  *choice = c;
}

// Group-limited top-k of one token from its scores and choices in shared memory.
template <int VPT>
__device__ __forceinline__ void route_grouped(const float* s_score, const float* s_choice, int E, int k, int n_group,
                                              int topk_group, int renorm, float scale, int lane, int* s_ids,
                                              float* __restrict__ out_w, int32_t* __restrict__ out_ids) {
  float key[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int e = lane + 32 * i;
    key[i] = (e < E) ? s_choice[e] : kNegInf;
  }
  // group score: sum of the two largest choices of the group.  The warp's lanes are shared out among the groups, as many to
  // each as the next power of two allows, and meet by shuffles (one lane per group: 32 dependent steps for 8 groups of 32).
  const int gsz = E / n_group;
  int per = 1;
  while (2 * per * n_group <= 32) per *= 2;
  const int group = lane / per;
  float m1 = kNegInf, m2 = kNegInf;
  if (group < n_group) {
    for (int i = lane % per; i < gsz; i += per) {
      const float c = s_choice[group * gsz + i];
      m2 = fmaxf(m2, fminf(m1, c));
      m1 = fmaxf(m1, c);
    }
  }
  for (int off = per >> 1; off > 0; off >>= 1) {
    const float o1 = __shfl_xor_sync(0xffffffffu, m1, off), o2 = __shfl_xor_sync(0xffffffffu, m2, off);
    m2 = fmaxf(fminf(m1, o1), fmaxf(m2, o2));
    m1 = fmaxf(m1, o1);
  }
  float gscore = (gsz >= 2) ? (m1 + m2) : m1;
  if (gscore != gscore) gscore = kNegInf;  // +inf + -inf
  gscore = __shfl_sync(0xffffffffu, gscore, min(lane, n_group - 1) * per);  // lane g: group g
  if (lane >= n_group) gscore = kNegInf;
  // keep the topk_group best groups (ties -> lower group index)
  uint32_t keep = 0;
  for (int j = 0; j < topk_group; ++j) {
    const bool open = lane < n_group && !((keep >> lane) & 1u);
    const int g = warp_argmax(open ? ordered_bits(gscore) : 0u, open ? lane : 0x7fffffff);
    if (g < 32) keep |= 1u << g;
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int e = lane + 32 * i;
    if (e < E && !((keep >> (e / gsz)) & 1u)) key[i] = kNegInf;
  }
  select_topk<VPT>(key, E, k, lane, s_ids);
  __syncwarp();
  int id = (lane < k) ? min(max(s_ids[lane], 0), E - 1) : 0;
  float w = (lane < k) ? s_score[id] : 0.f;
  if (renorm) {
    float s = 0.f;
    for (int j = 0; j < k; ++j) s += __shfl_sync(0xffffffffu, w, j);
    w = __fdiv_rn(w, s + 1e-20f);
  }
  w *= scale;
  if (lane < k) {
    out_w[lane] = w;
    out_ids[lane] = id;
  }
}
#endif

}  // namespace fmoe
