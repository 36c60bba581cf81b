// Row-wise helper kernels around the grouped GEMMs (all HBM-bound, 16-byte accesses):
//   fmoe_quant_fp8_group128 : per-row, per-128-channel e4m3 quantisation (+ optional row gather)
//   fmoe_gather_rows        : copy rows into the padded expert-sorted order
//   fmoe_moe_sum            : out[t] = sum_j z[t,j], optional post-scale
#include "rows.cuh"

#include <type_traits>

namespace fmoe {
namespace {

enum class RowMode { kMap, kScatter, kInPlace, kExpert };

// Source row of output position p: p itself without a map; with a map, the map's entry divided by map_div,
// or p when map_div is 0 (the map then only marks padding).  -1 = padding position.
__device__ __forceinline__ int64_t mapped_row(const int32_t* row_map, int map_div, int64_t sentinel, int64_t p) {
  if (!row_map) return p;
  int32_t s = row_map[p];
  if (s < 0 || (int64_t)s >= sentinel) return -1;
  return map_div ? s / map_div : p;
}


// The work is the flat list of (output row, 128-channel group) items; 16 lanes own one item: each lane loads
// 8 consecutive channels (16 bytes of bf16, 32 of fp32) and writes 8 bytes.  A 16-lane team walks the list with
// the grid's team count as stride and loads kIlp items before it reduces any, so that short rows (few groups)
// keep as many loads in flight as long ones.  Row and group of an item advance by a fixed step: no division
// inside the loop.
// With `pos` (position of every slot in the expert-sorted order) the layer walks what is there instead of the padded order,
// most of which is padding when experts have few rows:
//   RowMode::kInPlace : row p is slot p; the row at its position is quantised into the same position
//   RowMode::kExpert  : blockIdx.y is an expert, its rows start at map_div times that and go to its positions; experts with
//                       more than map_div rows are left out.  `pos` is the expert table (first row [E], rows [E], ..)
// DeepSeek-V3, 128 tokens (1024 rows in 21k positions): 26 -> 10 us before the gate/up GEMM, 38 -> 7 us before the down GEMM;
// 2048 tokens with one scale per row: 67 -> 42 us.
template <typename InT, RowMode MODE>
__global__ void __launch_bounds__(256)
quant_group128_kernel(const InT* __restrict__ x, int64_t rows_out, int64_t K, const int32_t* __restrict__ row_map,
                      int map_div, int64_t sentinel, const int32_t* __restrict__ num_rows_dev,
                      uint8_t* __restrict__ q, float* __restrict__ scale, const int32_t* __restrict__ pos) {
  if constexpr (MODE == RowMode::kMap) pdl_entry();
  else pdl_entry_late();
  constexpr int kIlp = 4;
  const int sub = threadIdx.x & 15;  // lane inside the 16-lane team
  const int groups = (int)(K / 128);
  int64_t limit = num_rows_dev ? min((int64_t)*num_rows_dev, rows_out) : rows_out;
  int64_t base = 0;
  if constexpr (MODE == RowMode::kExpert) {
    base = pos[blockIdx.y];
    limit = pos[gridDim.y + blockIdx.y];
    if (limit > map_div) return;
  }
  const int64_t teams = (int64_t)gridDim.x * 16;
  const int64_t team = (int64_t)blockIdx.x * 16 + (threadIdx.x >> 4);
  const int64_t step_p = teams / groups;
  const int step_g = (int)(teams % groups);
  int64_t p = team / groups;  // item of this team: (row p, group g); the next one is `teams` items further
  int g = (int)(team % groups);
  while (__any_sync(0xffffffffu, p < limit)) {  // the warp stays together: shuffles of half a warp each take their own turn
    float v[kIlp][8];
    int64_t pu[kIlp];
    int gu[kIlp];
    bool real[kIlp];
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      pu[u] = p;
      gu[u] = g;
      real[u] = false;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[u][i] = 0.f;
      if (p < limit) {
        const int64_t r = MODE == RowMode::kExpert ? (int64_t)blockIdx.y * map_div + p
                          : (MODE == RowMode::kInPlace ? pos[p] : mapped_row(row_map, map_div, sentinel, p));
        if constexpr (MODE == RowMode::kExpert) pu[u] = base + p;
        if constexpr (MODE == RowMode::kInPlace) pu[u] = r;
        real[u] = r >= 0;
        if (r >= 0) {
          const InT* src = x + r * K + g * 128 + sub * 8;
          if constexpr (sizeof(InT) == 4) {
            float4 f0 = __ldg(reinterpret_cast<const float4*>(src));
            float4 f1 = __ldg(reinterpret_cast<const float4*>(src) + 1);
            v[u][0] = f0.x; v[u][1] = f0.y; v[u][2] = f0.z; v[u][3] = f0.w;
            v[u][4] = f1.x; v[u][5] = f1.y; v[u][6] = f1.z; v[u][7] = f1.w;
          } else {
            uint4 raw = __ldg(reinterpret_cast<const uint4*>(src));
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              v[u][2 * i] = __low2float(h[i]);
              v[u][2 * i + 1] = __high2float(h[i]);
            }
          }
        }
      }
      p += step_p;
      g += step_g;
      if (g >= groups) {
        g -= groups;
        ++p;
      }
    }
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[u][i]));
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
      if constexpr (MODE != RowMode::kMap) {
        if (!real[u]) continue;
      } else if (pu[u] >= limit) {  // uniform over the 16 lanes of the team
        continue;
      }
      uint2* dst = reinterpret_cast<uint2*>(q + pu[u] * K + (int64_t)gu[u] * 128 + sub * 8);
      if (!real[u]) {  // padding position: zeros with a unit scale
        *dst = make_uint2(0, 0);
        if (sub == 0) scale[pu[u] * groups + gu[u]] = 1.0f;
        continue;
      }
      const float s = group_scale(amax);
      const uint2 bytes = quant8(v[u], s, __frcp_rn(s), amax <= 3.0e38f);
      *dst = bytes;
      if (sub == 0) scale[pu[u] * groups + gu[u]] = s;
    }
  }
}

// Token rows quantised once and stored at the positions of their k slots, scales by token.  Eight lanes own a group of 128
// channels, 32 bytes each, and store 16: most of what this kernel does is storing, and its stores bound it (sixteen lanes and
// 8-byte stores, shuffles by half warps: DeepSeek-V3, 4096 tokens, 70 us; this one 47 us).
__global__ void __launch_bounds__(256)
quant_scatter128_kernel(const __nv_bfloat16* __restrict__ x, int64_t T, int64_t K, int k, const int32_t* __restrict__ pos,
                        uint8_t* __restrict__ q, float* __restrict__ scale) {
  pdl_entry_late();
  constexpr int kIlp = 2;
  const int sub = threadIdx.x & 7;
  const int groups = (int)(K / 128);
  const int64_t teams = (int64_t)gridDim.x * 32, team = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  const int64_t step_p = teams / groups;
  const int step_g = (int)(teams % groups);
  int64_t p = team / groups;  // item of this team: (token p, group g); the next one is `teams` items further
  int g = (int)(team % groups);
  while (__any_sync(0xffffffffu, p < T)) {  // the warp stays together for its shuffles
    uint4 raw[kIlp][2];
    int64_t pu[kIlp];
    int gu[kIlp];
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      pu[u] = p;
      gu[u] = g;
      raw[u][0] = raw[u][1] = make_uint4(0, 0, 0, 0);
      if (p < T) {
        const uint4* src = reinterpret_cast<const uint4*>(x + p * K + g * 128 + sub * 16);
        raw[u][0] = __ldg(src);
        raw[u][1] = __ldg(src + 1);
      }
      p += step_p;
      g += step_g;
      if (g >= groups) {
        g -= groups;
        ++p;
      }
    }
#pragma unroll
    for (int u = 0; u < kIlp; ++u) {
      float v[2][8], amax = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&raw[u][h]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[h][2 * i] = __low2float(e[i]);
          v[h][2 * i + 1] = __high2float(e[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[h][i]));
      }
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
      if (pu[u] >= T) continue;
      const float s = group_scale(amax), r = __frcp_rn(s);
      const uint2 lo = quant8(v[0], s, r, amax <= 3.0e38f), hi = quant8(v[1], s, r, amax <= 3.0e38f);
      uint8_t* at = q + (int64_t)gu[u] * 128 + sub * 16;
      for (int j = 0; j < k; ++j) {
        const int32_t to = pos[pu[u] * k + j];
        if (to >= 0) *reinterpret_cast<uint4*>(at + (int64_t)to * K) = make_uint4(lo.x, lo.y, hi.x, hi.y);
      }
      if (sub == 0) scale[pu[u] * groups + gu[u]] = s;
    }
  }
}

// Per-token dynamic quantisation to e4m3 with ONE scale per row (the activation side of per-channel w8a8).  A team of
// TEAM threads (a warp for rows up to 4096 channels, the whole CTA above) owns an output row and holds it in
// registers between the amax pass and the conversion: VECS 16-byte vectors per thread.  scale = max(amax / 448,
// 1 / (448 * 512)), q = rne(x / scale) saturated: the rule of vLLM's dynamic per-token quantiser.  Row modes as above.
template <int TEAM, int VECS, RowMode MODE>
__global__ void __launch_bounds__(256)
quant_row_kernel(const __nv_bfloat16* __restrict__ x, int64_t rows_out, int64_t K, const int32_t* __restrict__ row_map,
                 int map_div, int64_t sentinel, const int32_t* __restrict__ num_rows_dev, uint8_t* __restrict__ q,
                 float* __restrict__ scale, const int32_t* __restrict__ pos) {
  if constexpr (MODE == RowMode::kMap) pdl_entry();
  else pdl_entry_late();
  __shared__ float s_max[8];
  constexpr int kTeams = 256 / TEAM;
  const int lane = threadIdx.x % TEAM;
  const int64_t limit = num_rows_dev ? min((int64_t)*num_rows_dev, rows_out) : rows_out;
  const int vecs = (int)(K / 8);  // 16-byte vectors per row
  // p is the same for all threads of a team (TEAM == 256: of the CTA, so the __syncthreads below are uniform)
  for (int64_t p = (int64_t)blockIdx.x * kTeams + threadIdx.x / TEAM; p < limit; p += (int64_t)gridDim.x * kTeams) {
    const int64_t r = MODE == RowMode::kScatter ? p : (MODE == RowMode::kInPlace ? pos[p] : mapped_row(row_map, map_div, sentinel, p));
    const int64_t to_row = MODE == RowMode::kInPlace ? r : p;
    uint2* dst = reinterpret_cast<uint2*>(q + to_row * K);
    if (r < 0) {  // padding position: zeros with a unit scale
      for (int c = lane; c < vecs; c += TEAM) dst[c] = make_uint2(0, 0);
      if (lane == 0) scale[p] = 1.0f;
      continue;
    }
    const uint4* src = reinterpret_cast<const uint4*>(x + r * K);
    int32_t to[8];  // kScatter: the first slots' positions, fetched with the row (2048 tokens x 7168: 28 -> 21 us)
    if constexpr (MODE == RowMode::kScatter) {
#pragma unroll
      for (int j = 0; j < 8; ++j) to[j] = j < map_div ? pos[p * map_div + j] : -1;
    }
    uint4 raw[VECS];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int c = lane + i * TEAM;
      raw[i] = make_uint4(0, 0, 0, 0);
      if (c < vecs) {
        raw[i] = __ldg(src + c);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fmaxf(fabsf(__low2float(h[j])), fabsf(__high2float(h[j]))));
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    if constexpr (TEAM == 256) {
      __syncthreads();  // s_max of the previous row has been read by everyone
      if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = amax;
      __syncthreads();
      amax = s_max[0];
#pragma unroll
      for (int w = 1; w < 8; ++w) amax = fmaxf(amax, s_max[w]);
    }
    const float s = fmaxf(__fdiv_rn(amax, 448.0f), 1.0f / (448.0f * 512.0f));
    const float rcp = __frcp_rn(s);
    const bool finite = amax <= 3.0e38f;
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int c = lane + i * TEAM;
      if (c >= vecs) continue;
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i]);
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] = __low2float(h[j]);
        v[2 * j + 1] = __high2float(h[j]);
      }
      const uint2 bytes = quant8(v, s, rcp, finite);
      if constexpr (MODE == RowMode::kScatter) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (to[j] >= 0) reinterpret_cast<uint2*>(q + (int64_t)to[j] * K)[c] = bytes;
        for (int j = 8; j < map_div; ++j) {
          const int32_t further = pos[p * map_div + j];
          if (further >= 0) reinterpret_cast<uint2*>(q + (int64_t)further * K)[c] = bytes;
        }
      } else {
        dst[c] = bytes;
      }
    }
    if (lane == 0) scale[to_row] = s;
  }
}

// A warp per output row, eight 16-byte loads per lane in flight, the next row's map entry fetched ahead: 16384 rows of 4 KB
// and 65536 of 4 KB went from 2.8 to about 5 TB/s against a CTA per row with one load per thread.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ x, int64_t rows_out, int64_t vec_per_row,
                   const int32_t* __restrict__ row_map, int map_div, int64_t sentinel,
                   const int32_t* __restrict__ num_rows_dev, uint4* __restrict__ out) {
  pdl_entry();
  constexpr int kIlp = 8;
  const int lane = threadIdx.x & 31;
  const int64_t limit = num_rows_dev ? min((int64_t)*num_rows_dev, rows_out) : rows_out;
  const int64_t stride = (int64_t)gridDim.x * 8;
  int64_t p = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  int64_t r = p < limit ? mapped_row(row_map, map_div, sentinel, p) : -1;
  for (; p < limit; p += stride) {
    const int64_t next = p + stride < limit ? mapped_row(row_map, map_div, sentinel, p + stride) : -1;
    const uint4* src = x + r * vec_per_row;
    uint4* dst = out + p * vec_per_row;
    for (int64_t c0 = lane; c0 < vec_per_row; c0 += 32 * kIlp) {
      uint4 v[kIlp];
#pragma unroll
      for (int i = 0; i < kIlp; ++i) {
        const int64_t c = c0 + 32 * i;
        v[i] = (r >= 0 && c < vec_per_row) ? __ldg(src + c) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < kIlp; ++i) {
        const int64_t c = c0 + 32 * i;
        if (c < vec_per_row) dst[c] = v[i];
      }
    }
    r = next;
  }
}

// Every token row to the positions of its k slots: read once, k stores (Qwen3, 7777 tokens: 64 -> 46 us, 5.9 TB/s of
// stores).  A warp per 2 KB piece of a row, so that few long rows still fill the chip.
__global__ void __launch_bounds__(256)
scatter_rows_kernel(const uint4* __restrict__ x, int64_t T, int k, int vec_per_row, int pieces, const int32_t* __restrict__ pos,
                    uint4* __restrict__ out) {
  pdl_entry_late();
  constexpr int kIlp = 4;
  const int lane = threadIdx.x & 31;
  const int64_t items = T * pieces;
  for (int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); i < items; i += (int64_t)gridDim.x * 8) {
    const int64_t t = i / pieces;
    const int c0 = (int)(i % pieces) * 32 * kIlp + lane;
    const int32_t my_pos = lane < k ? pos[t * k + lane] : -1;
    uint4 v[kIlp];
#pragma unroll
    for (int u = 0; u < kIlp; ++u)
      if (c0 + 32 * u < vec_per_row) v[u] = __ldg(x + t * vec_per_row + c0 + 32 * u);
    for (int j = 0; j < k; ++j) {
      const int32_t to = j < 32 ? __shfl_sync(0xffffffffu, my_pos, j) : pos[t * k + j];
      if (to < 0) continue;
      uint4* dst = out + (int64_t)to * vec_per_row;
#pragma unroll
      for (int u = 0; u < kIlp; ++u)
        if (c0 + 32 * u < vec_per_row) dst[c0 + 32 * u] = v[u];
    }
  }
}

// each thread owns 8 bf16 (or 4 f32) columns of one token and adds the k slots in order; kIlp slots' loads are issued
// before the first is added.  HBM bounds it from a few MB on: 4096 tokens x 8 slots x 7168 94.7 -> 78.4 us (6.7 TB/s) with
// eight loads in flight instead of four and 32-bit indices, 7777 x 8 x 2048 53.1 -> 43.0 us, 1024 x 8 x 1280 7.8 -> 6.0 us.
template <typename T, int kIlp, typename Index>
__global__ void __launch_bounds__(256, kIlp <= 2 ? 8 : 4)
moe_sum_kernel(const T* __restrict__ z, int64_t Tn, int k, int64_t H, float scale, const T* __restrict__ addend,
               T* __restrict__ out) {
  pdl_entry();
  constexpr int V = 16 / sizeof(T);
  const Index vec_per_row = (Index)(H / V);
  const Index total = (Index)(Tn * vec_per_row);
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (Index)gridDim.x * blockDim.x) {
    const Index row = i / vec_per_row, c = i - row * vec_per_row;
    const int64_t t = row;
    const uint4* src = reinterpret_cast<const uint4*>(z + t * k * H) + c;
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.f;
    for (int j0 = 0; j0 < k; j0 += kIlp) {
      uint4 raw[kIlp];
#pragma unroll
      for (int j = 0; j < kIlp; ++j)
        if (j0 + j < k) raw[j] = __ldg(src + (int64_t)(j0 + j) * vec_per_row);
#pragma unroll
      for (int j = 0; j < kIlp; ++j) {
        if (j0 + j < k) {
          const T* e = reinterpret_cast<const T*>(&raw[j]);
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] += to_f32(e[v]);
        }
      }
    }
    uint4 res;
    T* o = reinterpret_cast<T*>(&res);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      T r = from_f32<T>(acc[v]);
      if (scale != 1.0f) r = from_f32<T>(to_f32(r) * scale);
      o[v] = r;
    }
    if (addend) {  // e.g. the shared expert's output: one more rounded add, as the separate `+=` would do
      uint4 raw = __ldg(reinterpret_cast<const uint4*>(addend + t * H) + c);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int v = 0; v < V; ++v) o[v] = from_f32<T>(to_f32(o[v]) + to_f32(e[v]));
    }
    reinterpret_cast<uint4*>(out + t * H)[c] = res;
  }
}

}  // namespace
}  // namespace fmoe

extern "C" int fmoe_quant_fp8_group128(const void* x, int in_dtype, int64_t rows_out, int64_t K,
                                       const int32_t* row_map, int map_div, int64_t map_sentinel,
                                       const int32_t* num_rows_dev, void* q, float* scale, void* stream) {
  using namespace fmoe;
  auto st = (cudaStream_t)stream;
  FMOE_REQUIRE(K > 0 && K % 128 == 0, "quant_fp8_group128: K must be a positive multiple of 128 (got %lld)", (long long)K);
  FMOE_REQUIRE(in_dtype == FMOE_BF16 || in_dtype == FMOE_F32, "quant_fp8_group128: in_dtype must be bf16 or f32");
  FMOE_REQUIRE(!row_map || map_div >= 0, "quant_fp8_group128: map_div must be >= 0");
  if (rows_out <= 0) return FMOE_OK;
  FMOE_REQUIRE(x && q && scale, "quant_fp8_group128: null pointer");
  FMOE_REQUIRE(aligned16(x) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0, "quant_fp8_group128: misaligned pointer");
  // 16 teams per CTA, 4 items per team and pass
  unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div<int64_t>(rows_out * (K / 128), 64), 148 * 8));
  if (in_dtype == FMOE_BF16)
    launch_pdl(quant_group128_kernel<__nv_bfloat16, RowMode::kMap>, dim3(grid), dim3(256), 0, st, (const __nv_bfloat16*)x, rows_out, K,
               row_map, map_div, map_sentinel, num_rows_dev, (uint8_t*)q, scale, nullptr);
  else
    launch_pdl(quant_group128_kernel<float, RowMode::kMap>, dim3(grid), dim3(256), 0, st, (const float*)x, rows_out, K, row_map,
               map_div, map_sentinel, num_rows_dev, (uint8_t*)q, scale, nullptr);
  return launch_status("quant_group128_kernel");
}

extern "C" int fmoe_quant_fp8_per_token(const void* x, int in_dtype, int64_t rows_out, int64_t K,
                                        const int32_t* row_map, int map_div, int64_t map_sentinel,
                                        const int32_t* num_rows_dev, void* q, float* scale, void* stream) {
  using namespace fmoe;
  auto st = (cudaStream_t)stream;
  FMOE_REQUIRE(K > 0 && K % 8 == 0 && K <= 16384, "quant_fp8_per_token: K must be a multiple of 8 up to 16384 (got %lld)",
               (long long)K);
  FMOE_REQUIRE(in_dtype == FMOE_BF16, "quant_fp8_per_token: in_dtype must be bf16");
  FMOE_REQUIRE(!row_map || map_div >= 0, "quant_fp8_per_token: map_div must be >= 0");
  if (rows_out <= 0) return FMOE_OK;
  FMOE_REQUIRE(x && q && scale, "quant_fp8_per_token: null pointer");
  FMOE_REQUIRE(aligned16(x) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0, "quant_fp8_per_token: misaligned pointer");
  auto go = [&](auto kernel, int teams) {
    unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(rows_out, teams), 148 * 8);
    launch_pdl(kernel, dim3(grid), dim3(256), 0, st, (const __nv_bfloat16*)x, rows_out, K, row_map, map_div, map_sentinel,
               num_rows_dev, (uint8_t*)q, scale, nullptr);
  };
  if (K <= 2048) go(quant_row_kernel<32, 8, RowMode::kMap>, 8);         // a warp per row, 8 rows per CTA
  else if (K <= 4096) go(quant_row_kernel<32, 16, RowMode::kMap>, 8);
  else go(quant_row_kernel<256, 8, RowMode::kMap>, 1);                  // a CTA per row
  return launch_status("quant_row_kernel");
}

int fmoe::run_scatter_rows(const void* x, int elem_bytes, int64_t T, int k, int64_t K, const int32_t* slot_pos, void* out,
                           cudaStream_t st) {
  FMOE_REQUIRE((K * elem_bytes) % 16 == 0 && K * elem_bytes < (1ll << 31), "scatter_rows: row size must be a multiple of 16 bytes");
  FMOE_REQUIRE(x && out && aligned16(x) && aligned16(out), "scatter_rows: null or misaligned pointer");
  const int vecs = (int)(K * elem_bytes / 16), pieces = ceil_div(vecs, 128);
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(T * pieces, 8), 148 * 8);
  launch_pdl(scatter_rows_kernel, dim3(grid), dim3(256), 0, st, (const uint4*)x, T, k, vecs, pieces, slot_pos, (uint4*)out);
  return launch_status("scatter_rows_kernel");
}

int fmoe::run_quant_scatter(const void* x, int64_t T, int k, int64_t K, const int32_t* slot_pos, bool per_row, void* q,
                            float* scale, cudaStream_t st) {
  FMOE_REQUIRE(K > 0 && K % (per_row ? 8 : 128) == 0 && (!per_row || K <= 16384), "quant_scatter: bad K %lld", (long long)K);
  FMOE_REQUIRE(x && q && scale && aligned16(x) && aligned16(q), "quant_scatter: null or misaligned pointer");
  auto go = [&](auto kernel, int64_t ctas) {
    launch_pdl(kernel, dim3((unsigned)std::min<int64_t>(std::max<int64_t>(ctas, 1), 148 * 8)), dim3(256), 0, st,
               (const __nv_bfloat16*)x, T, K, nullptr, k, 0, nullptr, (uint8_t*)q, scale, slot_pos);
  };
  if (!per_row) {
    const int64_t ctas = std::min<int64_t>(std::max<int64_t>(ceil_div<int64_t>(T * (K / 128), 64), 1), 148 * 8);
    launch_pdl(quant_scatter128_kernel, dim3((unsigned)ctas), dim3(256), 0, st, (const __nv_bfloat16*)x, T, K, k, slot_pos, (uint8_t*)q,
               scale);
  } else if (K <= 2048) go(quant_row_kernel<32, 8, RowMode::kScatter>, ceil_div<int64_t>(T, 8));
  else if (K <= 4096) go(quant_row_kernel<32, 16, RowMode::kScatter>, ceil_div<int64_t>(T, 8));
  else go(quant_row_kernel<256, 8, RowMode::kScatter>, T);
  return launch_status("quant_scatter");
}

int fmoe::run_quant_rows(const void* x, int64_t numel, int64_t K, const int32_t* slot_pos, void* q, float* scale, cudaStream_t st) {
  FMOE_REQUIRE(K > 0 && K % 8 == 0 && K <= 16384, "quant_rows: bad K %lld", (long long)K);
  FMOE_REQUIRE(x && q && scale && aligned16(x) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0, "quant_rows: null or misaligned pointer");
  auto go = [&](auto kernel, int64_t ctas) {
    launch_pdl(kernel, dim3((unsigned)std::min<int64_t>(std::max<int64_t>(ctas, 1), 148 * 8)), dim3(256), 0, st,
               (const __nv_bfloat16*)x, numel, K, nullptr, 1, 0, nullptr, (uint8_t*)q, scale, slot_pos);
  };
  if (K <= 2048) go(quant_row_kernel<32, 8, RowMode::kInPlace>, ceil_div<int64_t>(numel, 8));
  else if (K <= 4096) go(quant_row_kernel<32, 16, RowMode::kInPlace>, ceil_div<int64_t>(numel, 8));
  else go(quant_row_kernel<256, 8, RowMode::kInPlace>, numel);
  return launch_status("quant_rows");
}

int fmoe::run_quant_slots(const float* x, int64_t numel, int64_t K, const int32_t* slot_pos, void* q, float* scale, cudaStream_t st) {
  FMOE_REQUIRE(K > 0 && K % 128 == 0, "quant_slots: bad K %lld", (long long)K);
  FMOE_REQUIRE(x && q && scale && aligned16(x) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0, "quant_slots: null or misaligned pointer");
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(numel * (K / 128), 64), 148 * 8);
  launch_pdl(quant_group128_kernel<float, RowMode::kInPlace>, dim3(grid), dim3(256), 0, st, x, numel, K, nullptr, 1, 0, nullptr,
             (uint8_t*)q, scale, slot_pos);
  return launch_status("quant_slots");
}

int fmoe::run_quant_experts(const float* x, int64_t numel, int64_t K, int num_experts, const int32_t* table, int max_rows, void* q,
                            float* scale, cudaStream_t st) {
  FMOE_REQUIRE(K > 0 && K % 128 == 0, "quant_experts: bad K %lld", (long long)K);
  FMOE_REQUIRE(x && q && scale && aligned16(x) && (reinterpret_cast<uintptr_t>(q) & 7u) == 0, "quant_experts: null or misaligned pointer");
  // 64 items per CTA and pass; as many CTAs per expert as its rows on average (at most max_rows) ask for
  const int64_t rows = std::min<int64_t>(ceil_div<int64_t>(numel, num_experts), max_rows);
  const unsigned per_expert = (unsigned)std::min<int64_t>(std::max<int64_t>(1, rows * (K / 128) / 128), 8);
  launch_pdl(quant_group128_kernel<float, RowMode::kExpert>, dim3(per_expert, num_experts), dim3(256), 0, st, x, 0, K, nullptr,
             max_rows, 0, nullptr, (uint8_t*)q, scale, table);
  return launch_status("quant_experts");
}

extern "C" int fmoe_gather_rows(const void* x, int elem_bytes, int64_t rows_out, int64_t K,
                                const int32_t* row_map, int map_div, int64_t map_sentinel,
                                const int32_t* num_rows_dev, void* out, void* stream) {
  using namespace fmoe;
  auto st = (cudaStream_t)stream;
  FMOE_REQUIRE(elem_bytes == 2 || elem_bytes == 4 || elem_bytes == 1, "gather_rows: elem_bytes must be 1, 2 or 4");
  FMOE_REQUIRE(K > 0 && (K * elem_bytes) % 16 == 0, "gather_rows: row size must be a multiple of 16 bytes");
  FMOE_REQUIRE(row_map && map_div >= 1, "gather_rows: row_map required");
  if (rows_out <= 0) return FMOE_OK;
  FMOE_REQUIRE(x && out && aligned16(x) && aligned16(out), "gather_rows: null or misaligned pointer");
  unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(rows_out, 8), 148 * 8);
  launch_pdl(gather_rows_kernel, dim3(grid), dim3(256), 0, st, (const uint4*)x, rows_out, K * elem_bytes / 16, row_map,
             map_div, map_sentinel, num_rows_dev, (uint4*)out);
  return launch_status("gather_rows_kernel");
}

extern "C" int fmoe_moe_sum(const void* z, int dtype, int64_t T, int k, int64_t H, float scale, void* out,
                            void* stream) {
  return fmoe_moe_sum_add(z, dtype, T, k, H, scale, nullptr, out, stream);
}

extern "C" int fmoe_moe_sum_add(const void* z, int dtype, int64_t T, int k, int64_t H, float scale,
                                const void* addend, void* out, void* stream) {
  using namespace fmoe;
  FMOE_REQUIRE(dtype == FMOE_BF16 || dtype == FMOE_F32, "moe_sum: dtype must be bf16 or f32");
  const int eb = dtype == FMOE_BF16 ? 2 : 4;
  FMOE_REQUIRE(k >= 1 && H > 0 && (H * eb) % 16 == 0, "moe_sum: need k >= 1 and H*elem %% 16 == 0");
  if (T <= 0) return FMOE_OK;
  FMOE_REQUIRE(z && out && aligned16(z) && aligned16(out) && aligned16(addend), "moe_sum: null or misaligned pointer");
  int64_t total = T * (H * eb / 16);
  unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(total, 256), 148 * 16);
  auto st = (cudaStream_t)stream;
  auto go = [&](auto kernel, auto* zt) {
    using E = std::remove_pointer_t<decltype(zt)>;
    launch_pdl(kernel, dim3(grid), dim3(256), 0, st, (const E*)z, T, k, H, scale, (const E*)addend, (E*)out);
  };
  __nv_bfloat16* b16 = nullptr;
  float* f32 = nullptr;
  // as many loads in flight per thread as a token has slots, up to 8; two slots: more CTAs instead
  auto pick = [&](auto index) {
    using I = decltype(index);
    if (dtype == FMOE_BF16) {
      if (k <= 2) go(moe_sum_kernel<__nv_bfloat16, 2, I>, b16);
      else if (k <= 4) go(moe_sum_kernel<__nv_bfloat16, 4, I>, b16);
      else go(moe_sum_kernel<__nv_bfloat16, 8, I>, b16);
    } else {
      if (k <= 2) go(moe_sum_kernel<float, 2, I>, f32);
      else go(moe_sum_kernel<float, 4, I>, f32);
    }
  };
  if (total + (int64_t)grid * 256 < (1ll << 31)) pick(uint32_t{});  // 64-bit divisions would be a third of the instructions
  else pick(int64_t{});
  return launch_status("moe_sum_kernel");
}
