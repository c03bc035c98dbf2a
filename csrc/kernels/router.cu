// MoE top-k router, entirely on the device.
//
//   1. router_topk_kernel: logits[t, e] = x[t, :] . Wg[e, :] (fp32 accumulate), the k largest
//      logits per token (ties -> lower expert index) and their softmax over the selected k, which
//      equals "softmax over all experts, take top-k, renormalise" (what Mixtral does).
//   2. router_plan_kernel (one CTA): per-expert counts, exclusive offsets, and a stable position
//      for every (token, slot) pair in expert-sorted order:
//         row_of[t, j]    position of pair (t, j) in the sorted list
//         src_token[r]    token whose activation belongs at sorted row r
//      The pairs are walked in order with warp votes, so the layout is the same on every run and
//      on every rank.
// The grouped GEMM reads counts/offsets straight from device memory; nothing returns to the host.
//
// Replaces the reference's host-side routing (crates/skein_runtime/src/distributed/
// segment_runner.rs:249,1417: D2H of the router logits, host top-k softmax, pointer rebinding) and
// the graph-level iterative-argmax top_k_route (crates/skein_emit/src/op_wiring.rs:1667-1712).
#include "ptx.cuh"
#include "launch.cuh"
#include "route.cuh"
#include <cuda_bf16.h>
#include <math.h>

namespace skein {

constexpr int RT_MAX_E = 64;
constexpr int RT_MAX_K = 8;
constexpr int PLAN_WARPS = 16, PLAN_INTS = (PLAN_WARPS + 2) * RT_MAX_E + 1;

__device__ void router_plan_body(const int* __restrict__ expert_ids, int n_pairs, int E, int topk,
                                 int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ row_of,
                                 int* __restrict__ src_token, int e_first, int e_count, int* sh);

// The top-k of one token's logits, ties to the lower expert, and their softmax.
__device__ __forceinline__ void router_select(const float* z, int E, int topk, int* expert_ids, float* expert_w) {
  int ids[RT_MAX_K];
  float vals[RT_MAX_K];
  for (int j = 0; j < topk; ++j) {
    int best = -1;
    float bv = -INFINITY;
    for (int e = 0; e < E; ++e) {
      bool taken = false;
      for (int q = 0; q < j; ++q) taken |= (ids[q] == e);
      if (!taken && (best < 0 || z[e] > bv)) { best = e; bv = z[e]; }
    }
    ids[j] = best; vals[j] = bv;
  }
  float den = 0.f;
  const float vmax = vals[0];  // selections come out in descending order
  for (int j = 0; j < topk; ++j) { vals[j] = __expf(vals[j] - vmax); den += vals[j]; }
  for (int j = 0; j < topk; ++j) {
    expert_ids[j] = ids[j];
    expert_w[j] = vals[j] / den;
  }
}

// Counts a CTA whose choices are written (and fenced by their writers) in; true for the last one, which then sees all of them.
__device__ __forceinline__ bool router_last_cta(int* done_counter) {
  __shared__ int is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(done_counter, 1) == (int)gridDim.x - 1;
    if (is_last) *done_counter = 0;
  }
  __syncthreads();
  if (!is_last) return false;
  __threadfence();
  return true;
}

struct RouterOut {
  int* expert_ids;
  float *expert_w, *logits;
  int *counts, *offsets, *row_of, *src_token;
  int e_first, e_count;
  int* done_counter;
};

// Few tokens: grid = T, 512 threads: thread i owns 8 consecutive elements of the hidden vector per pass, so
// every load of a pass is issued before the first is consumed. The last CTA to finish also lays out
// the expert-sorted order (router_plan_body), which saves a launch on the decode path. Three CTAs per SM: with the layout's loads in flight the compiler
// took registers for two, and 300 tokens, a third round of CTAs, 16.0 instead of 13.5 us (4 experts x 8192).
__global__ void __launch_bounds__(512, 3) router_topk_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wg, int T, int H, int E,
                                                          int topk, const RouterOut o) {
  __shared__ float part[16][RT_MAX_E];
  __shared__ float logit[RT_MAX_E];
  __shared__ int plan_s[PLAN_INTS];
  const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e0 = 0; e0 < E; e0 += 8) {
    float a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = 0.f;
    for (int h = tid * 8; h < H; h += 512 * 8) {
      const uint4 xr = *reinterpret_cast<const uint4*>(x + (size_t)t * H + h);
      uint4 wr[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        wr[i] = (e0 + i < E) ? *reinterpret_cast<const uint4*>(wg + (size_t)(e0 + i) * H + h) : make_uint4(0, 0, 0, 0);
      const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&xr);
      float xf[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(xb[i]); xf[2 * i] = f.x; xf[2 * i + 1] = f.y; }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162* wb = reinterpret_cast<const __nv_bfloat162*>(&wr[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(wb[j]); a[i] += xf[2 * j] * f.x + xf[2 * j + 1] * f.y; }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float v = a[i];
      for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
      if (lane == 0 && e0 + i < E) part[warp][e0 + i] = v;
    }
  }
  __syncthreads();
  if (tid < E) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 16; ++w) v += part[w][tid];
    // the router projection is a bf16 linear layer: round like one
    logit[tid] = __bfloat162float(__float2bfloat16(v));
    if (o.logits) o.logits[(size_t)t * E + tid] = logit[tid];
  }
  __syncthreads();
  if (tid == 0) router_select(logit, E, topk, o.expert_ids + (size_t)t * topk, o.expert_w + (size_t)t * topk);
  if (o.done_counter == nullptr || !router_last_cta(o.done_counter)) return;
  router_plan_body(o.expert_ids, T * topk, E, topk, o.counts, o.offsets, o.row_of, o.src_token, o.e_first, o.e_count, plan_s);
}

// Many tokens: 16 of them x 8 experts are one mma.sync tile. What bounds it is the activations' bytes; with a CTA per token it was the router weights,
// fetched from L2 for every token (64 KB of them at 8 experts x 4096 for 8 KB of activations), and a chain of sums, selection and count per token. A
// CTA's 16 warps share the reduction dimension, 32 elements at a time: a lane's 16 bytes of a row are its part of two tiles (the order of the
// elements inside a tile is free as long as both operands use the same). 4096 tokens x 4096, 8 experts: 225 -> 20 us, 1000 tokens 38 -> 11.
constexpr int RR_TOKENS = 16;
__global__ void __launch_bounds__(512) router_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wg, int T, int H, int E,
                                                          int topk, const RouterOut o) {
  __shared__ float part[16][RR_TOKENS][8];
  __shared__ float logit[RR_TOKENS][RT_MAX_E + 1];
  __shared__ int plan_s[PLAN_INTS];
  const int t0 = blockIdx.x * RR_TOKENS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const __nv_bfloat16 *x0 = x + (size_t)min(t0 + g, T - 1) * H + c * 8, *x1 = x + (size_t)min(t0 + g + 8, T - 1) * H + c * 8;
  for (int e0 = 0; e0 < E; e0 += 8) {
    const __nv_bfloat16* w0 = wg + (size_t)min(e0 + g, E - 1) * H + c * 8;
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int h = warp * 32; h < H; h += 16 * 32) {
      const uint4 a = *reinterpret_cast<const uint4*>(x0 + h), b = *reinterpret_cast<const uint4*>(x1 + h), w = *reinterpret_cast<const uint4*>(w0 + h);
      auto mma = [&](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
      };
      mma(a.x, b.x, a.y, b.y, w.x, w.y);
      mma(a.z, b.z, a.w, b.w, w.z, w.w);
    }
    part[warp][g][2 * c] = d[0]; part[warp][g][2 * c + 1] = d[1];
    part[warp][g + 8][2 * c] = d[2]; part[warp][g + 8][2 * c + 1] = d[3];
    __syncthreads();
    if (tid < RR_TOKENS * 8) {
      const int k = tid >> 3, e = e0 + (tid & 7);
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 16; ++w) v += part[w][k][tid & 7];
      if (e < E) {
        logit[k][e] = __bfloat162float(__float2bfloat16(v));      // rounded like a bf16 linear layer
        if (o.logits && t0 + k < T) o.logits[(size_t)(t0 + k) * E + e] = logit[k][e];
      }
    }
    __syncthreads();
  }
  if (lane == 0 && t0 + warp < T) {
    const size_t at = (size_t)(t0 + warp) * topk;
    router_select(logit[warp], E, topk, o.expert_ids + at, o.expert_w + at);
    __threadfence();
  }
  if (o.done_counter == nullptr || !router_last_cta(o.done_counter)) return;
  router_plan_body(o.expert_ids, T * topk, E, topk, o.counts, o.offsets, o.row_of, o.src_token, o.e_first, o.e_count, plan_s);
}

// Stable expert-sorted layout by one CTA of 16 warps: each warp takes a run of consecutive pairs, 32 at a time, in which the lanes of an expert find
// each other; the warps' counts per expert, summed up in order, are where their runs begin. (One warp per expert over all pairs is a chain of
// n_pairs / 32 loads, twice: most of the router's time at 8192 pairs.) Experts outside [e_first, e_first + e_count) get count 0 (expert
// parallelism: not ours) and their pairs row -1.
__device__ void router_plan_body(const int* __restrict__ expert_ids, int n_pairs, int E, int topk,
                                 int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ row_of,
                                 int* __restrict__ src_token, int e_first, int e_count, int* sh) {
  int* at = sh;                               // [warps][RT_MAX_E]: counts, then next positions
  int* cnt_s = sh + PLAN_WARPS * RT_MAX_E;    // [RT_MAX_E]
  int* off_s = cnt_s + RT_MAX_E;              // [RT_MAX_E + 1]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int run = ((n_pairs + PLAN_WARPS - 1) / PLAN_WARPS + 31) / 32 * 32, lo = warp * run, hi = min(n_pairs, lo + run);
  constexpr int AHEAD = 8;                    // loads in flight per lane
  auto each = [&](auto take) {
    for (int i0 = lo; i0 < hi; i0 += 32 * AHEAD) {
      int id[AHEAD];
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        const int i = i0 + k * 32 + lane;
        id[k] = i < hi ? __ldcg(expert_ids + i) : -1;
        if (id[k] >= E) id[k] = -1;
      }
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        const unsigned same = __match_any_sync(0xffffffffu, id[k]);
        take(i0 + k * 32 + lane, id[k], same, lane == __ffs(same) - 1);
        __syncwarp();
      }
    }
  };
  for (int i = tid; i < PLAN_WARPS * RT_MAX_E; i += PLAN_WARPS * 32) at[i] = 0;
  __syncthreads();
  each([&](int, int e, unsigned same, bool leader) {
    if (e >= 0 && leader) at[warp * RT_MAX_E + e] += __popc(same);
  });
  __syncthreads();
  if (tid < E) {
    int c = 0;
    for (int w = 0; w < PLAN_WARPS; ++w) c += at[w * RT_MAX_E + tid];
    cnt_s[tid] = (tid >= e_first && tid < e_first + e_count) ? c : 0;
  }
  __syncthreads();
  if (tid == 0) {
    int a = 0;
    for (int e = 0; e < E; ++e) { off_s[e] = a; a += cnt_s[e]; }
    off_s[E] = a;
  }
  __syncthreads();
  if (tid < E) {
    counts[tid] = cnt_s[tid];
    offsets[tid] = off_s[tid];
    int a = off_s[tid];
    for (int w = 0; w < PLAN_WARPS; ++w) {
      const int c = at[w * RT_MAX_E + tid];
      at[w * RT_MAX_E + tid] = a;
      a += c;
    }
  }
  if (tid == 0) offsets[E] = off_s[E];  // total rows
  __syncthreads();
  each([&](int i, int e, unsigned same, bool leader) {
    int first = 0;
    if (e >= 0) first = at[warp * RT_MAX_E + e];
    __syncwarp();
    if (e < 0) return;
    if (cnt_s[e] > 0) {
      const int r = first + __popc(same & ((1u << lane) - 1));
      row_of[i] = r;
      src_token[r] = i / topk;
    } else {
      row_of[i] = -1;
    }
    if (leader) at[warp * RT_MAX_E + e] = first + __popc(same);
  });
}

__global__ void __launch_bounds__(PLAN_WARPS * 32) router_plan_kernel(const int* __restrict__ expert_ids, int n_pairs, int E,
                                                                      int topk, int* __restrict__ counts, int* __restrict__ offsets,
                                                                      int* __restrict__ row_of, int* __restrict__ src_token,
                                                                      int e_first, int e_count) {
  __shared__ int plan_s[PLAN_INTS];
  router_plan_body(expert_ids, n_pairs, E, topk, counts, offsets, row_of, src_token, e_first, e_count, plan_s);
}

// ---- group-limited selection over given logits, and a layout kernel pair for prefill-sized batches -----------------
// One warp per token; logits fp32 [T, E].
constexpr int RG_MAX_E = 256;
__global__ void __launch_bounds__(128) route_select_kernel(const float* __restrict__ logits, int T, int E, int topk, const SkeinRouteRule rule,
                                                           int* __restrict__ expert_ids, float* __restrict__ expert_w) {
  __shared__ float z[4][RG_MAX_E];
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * 4 + warp;
  if (t >= T) return;
  for (int e = lane; e < E; e += 32) z[warp][e] = logits[(size_t)t * E + e];
  __syncwarp();
  select_grouped_warp<RG_MAX_E>(z[warp], E, topk, rule, expert_ids + (size_t)t * topk, expert_w + (size_t)t * topk);
}

// Stable expert-sorted layout with one CTA per expert: the first kernel counts, the second derives its expert's offset from
// all counts and hands out positions chunk by chunk (256 pairs per chunk, warp ballots inside).
__global__ void __launch_bounds__(256) plan_count_kernel(const int* __restrict__ expert_ids, int n_pairs, int* __restrict__ counts) {
  __shared__ int sh[8];
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x;
  int c = 0;
  for (int i = threadIdx.x; i < n_pairs; i += 256) c += expert_ids[i] == e;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int a = 0;
    for (int w = 0; w < 8; ++w) a += sh[w];
    counts[e] = a;
  }
}
__global__ void __launch_bounds__(256) plan_place_kernel(const int* __restrict__ expert_ids, int n_pairs, int E, int topk,
                                                         const int* __restrict__ counts, int* __restrict__ offsets,
                                                         int* __restrict__ row_of, int* __restrict__ src_token) {
  __shared__ int wsum[8];
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int base = 0;
  for (int i = 0; i < e; ++i) base += counts[i];
  if (threadIdx.x == 0) {
    offsets[e] = base;
    if (e == E - 1) offsets[E] = base + counts[e];
  }
  for (int i0 = 0; i0 < n_pairs; i0 += 256) {
    const int i = i0 + threadIdx.x;
    const bool hit = i < n_pairs && expert_ids[i] == e;
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wsum[warp] = __popc(bal);
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) { if (w < warp) before += wsum[w]; total += wsum[w]; }
    if (hit) {
      const int r = base + before + __popc(bal & ((1u << lane) - 1));
      row_of[i] = r;
      src_token[r] = i / topk;
    }
    base += total;
    __syncthreads();
  }
}

}  // namespace skein

// Scores of E logits, group-limited top-k, weights (route.cuh: select_grouped_warp), then the expert-sorted layout.
extern "C" int skein_route_grouped(const float* logits, int T, int E, int topk, const SkeinRouteRule* rule, int* expert_ids, float* expert_w,
                                   int* counts, int* offsets, int* row_of, int* src_token, void* stream) {
  using namespace skein;
  if (T == 0) return 0;
  if (E > RG_MAX_E || !route_rule_ok(*rule, E, topk)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t rc = launch_pdl(route_select_kernel, dim3((T + 3) / 4), dim3(128), 0, s, logits, T, E, topk, *rule, expert_ids, expert_w);
  if (rc == cudaSuccess) rc = launch_pdl(plan_count_kernel, dim3(E), dim3(256), 0, s, (const int*)expert_ids, T * topk, counts);
  if (rc == cudaSuccess) rc = launch_pdl(plan_place_kernel, dim3(E), dim3(256), 0, s, (const int*)expert_ids, T * topk, E, topk, (const int*)counts, offsets, row_of, src_token);
  return (int)rc;
}

// With done_counter (a zeroed device int) the same launch also produces the expert-sorted layout
// (counts[E], offsets[E+1], row_of[T*topk], src_token[T*topk]); without it only ids and weights.
extern "C" int skein_router_topk(const void* x, const void* wg, int T, int H, int E, int topk, int* expert_ids,
                                 float* expert_w, float* logits_out, int* counts, int* offsets, int* row_of,
                                 int* src_token, int e_first, int e_count, int* done_counter, void* stream) {
  using namespace skein;
  if (T == 0) return 0;
  if (E > RT_MAX_E || topk > RT_MAX_K || topk > E || H % 8 != 0) return -1;
  const RouterOut o{expert_ids, expert_w, logits_out, counts, offsets, row_of, src_token, e_first, e_count, done_counter};
  const __nv_bfloat16 *xb = (const __nv_bfloat16*)x, *wb = (const __nv_bfloat16*)wg;
  // Few tokens are few tiles, and up to four experts leave half of a tile empty. CTA per token / tiles, us: 8 experts x 4096 15.5 / 13.1 at 256 tokens,
  // x 8192 19.4 / 17.6; 4 experts x 1024 8.5 / 7.9, x 8192 12.1 / 15.1, at 300 13.4 / 15.5, at 512 19.7 / 16.1.
  if (T >= 256 && H % 32 == 0 && (E > 4 || H <= 2048 || T >= 512)) router_rows_kernel<<<(T + RR_TOKENS - 1) / RR_TOKENS, 512, 0, (cudaStream_t)stream>>>(xb, wb, T, H, E, topk, o);
  else router_topk_kernel<<<T, 512, 0, (cudaStream_t)stream>>>(xb, wb, T, H, E, topk, o);
  return (int)cudaGetLastError();
}

extern "C" int skein_router_plan(const int* expert_ids, int n_pairs, int E, int topk, int* counts, int* offsets,
                                 int* row_of, int* src_token, int e_first, int e_count, void* stream) {
  using namespace skein;
  if (E > RT_MAX_E) return -1;
  router_plan_kernel<<<1, PLAN_WARPS * 32, 0, (cudaStream_t)stream>>>(expert_ids, n_pairs, E, topk, counts, offsets, row_of,
                                                                 src_token, e_first, e_count);
  return (int)cudaGetLastError();
}
