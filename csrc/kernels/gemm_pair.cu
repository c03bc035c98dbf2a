// Products of prefill chunks: Y[t, f] = sum_k X[t, k] * W[f, k] on pairs of CTAs (tcgen05 cta_group::2), optionally grouped.
//
// What bounds it: the tensor cores. With one CTA per tile, a 128 x 256 tile moves 48 KB into shared memory and reads 48 KB of it for every
// 512 cycles of MMAs, and a gate/up pair of 128 x 128 tiles more, which is above what shared memory delivers. A pair of CTAs on one
// 256 x 256 tile stages 32 KB per CTA for the same cycles: each holds half of the weight rows (M) and half of the token rows (N), and the
// MMA reads the other half of the tokens from its peer. Sums, order and precision are those of the streaming kernel (gemm_ws.cu).
//
//   * operands: weights are the M side (256 rows per pair; with a gate/up pair each CTA has 64 gate and the 64 matching up rows, so both
//     halves of an output meet in its tensor memory), tokens the N side: 32 .. 256 columns. A group's rows are cut into equal tiles of at most 256,
//     so a ragged group pads at most 31 rows per tile.
//   * order of the tiles: whole tiles are dealt in turn, so the pairs in flight work on neighbouring tiles of a band of RASTER feature tiles
//     and share their operands in L2 (equal contiguous shares of the line of all K-blocks, as the streaming kernel deals them, are far apart:
//     every CTA then streams its operands alone). The tiles of the last, incomplete round are cut along K among all pairs and come first;
//     their fp32 partials are parked in the workspace and summed in a fixed order by the epilogue warps while the MMAs go on.
//   * roles: warp 0 TMA producer, warp 1 MMA issuer (of the even CTA), warps 2-5 epilogue; two accumulators of 256 columns.
#include "gemm_ws.cuh"
#include "gemm_sched.cuh"
#include "ptx.cuh"
#include "launch.cuh"
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace skein {

int cached_tmap_2d_ld(CUtensorMap* out, const void* base, uint64_t rows, uint64_t k_elems, uint64_t ld, int elem_bytes, uint32_t box_rows);

constexpr int PAIR_THREADS = 192;
constexpr int PAIR_STAGES = 8;
constexpr int PAIR_ROWS = 128;                    // weight rows of one CTA's tile
constexpr int PAIR_COLS = 256;                    // tokens of a tile, at most
constexpr int PAIR_W_BYTES = PAIR_ROWS * 128;
constexpr int PAIR_XCH_FLOATS = 2 * 2 * 2 * 16 * 32;      // [buffer][warp pair][direction][column][lane]
constexpr int PAIR_SMEM_MAX = 223 * 1024;
constexpr int RASTER = 8;                         // feature tiles of a band: with 74 pairs in flight about 8 x 9 tiles share their operands

struct PairArgs {
  SkeinGemmParams p;
  int cap;                  // tokens of a tile, at most (a multiple of 32)
  int stages, x_box;        // x_box: token rows that one CTA's copy brings
  uint64_t budget_ns;
};

struct PairSched {
  int pre[SKEIN_MAX_GROUPS + 1], cnt[SKEIN_MAX_GROUPS], off[SKEIN_MAX_GROUPS], ntile[SKEIN_MAX_GROUPS], cols[SKEIN_MAX_GROUPS];
  int MT, KB, U;
  int R, split;      // the first R tiles are cut into `split` pieces along K: piece i of tile u is pair i * R + u's
  int halves;        // whole tiles are summed in two halves of K (see pair_sched)
};

// number of tiles of a group of c rows, and tokens per tile
__host__ __device__ __forceinline__ int pair_tiles(int c, int cap) { return (c + cap - 1) / cap; }
__host__ __device__ __forceinline__ int pair_cols(int c, int cap) {
  const int nt = pair_tiles(c, cap);
  return nt > 0 ? ((c + nt - 1) / nt + 31) / 32 * 32 : 32;
}
// Pieces that each tile of the last, incomplete round of R tiles is cut into along K (1: left whole). Whole, they idle the other pairs for
// KB K-blocks; cut, the parked partials cost about as much as 12 (512 rows, 4096 x 4096: 32.1 -> 27.0 us for 32 tiles of 64 K-blocks in two
// pieces; 512 rows, 2048 x 2048: 21.8 -> 17.3).
__host__ __device__ __forceinline__ int pair_split(int R, int KB, int pairs) {
  if (R == 0) return 1;
  int sp = pairs / R;
  sp = sp < 8 ? sp : 8;
  sp = sp < KB / 4 ? sp : KB / 4;
  return sp > 1 && KB - (KB + sp - 1) / sp > 12 ? sp : 1;
}

__device__ __forceinline__ void pair_sched(PairSched& s, const SkeinGemmParams& p, int cap, int pairs) {
  const int ft = p.mode == 1 ? PAIR_ROWS : 2 * PAIR_ROWS;
  s.MT = (p.F + ft - 1) / ft;
  s.KB = (p.K + 63) / 64;
  long long acc = 0;
  for (int g = 0; g < p.G; ++g) {
    const int c = p.group_cnt ? p.group_cnt[g] : p.t_static;
    s.off[g] = p.group_off ? p.group_off[g] : 0;
    s.cnt[g] = c;
    s.ntile[g] = c > 0 ? pair_tiles(c, cap) : 1;
    s.cols[g] = pair_cols(c, cap);
    s.pre[g] = (int)acc;
    acc += c > 0 ? (long long)s.MT * pair_tiles(c, cap) : 0;
  }
  if (acc * s.KB >= (1ll << 31)) {
    report_status(p.status, ST_BAD_INDEX, p.G);
    acc = 0;
  }
  s.pre[p.G] = s.U = (int)acc;
  s.split = pair_split(s.U % pairs, s.KB, pairs);
  s.R = s.split > 1 ? s.U % pairs : 0;
  // Outputs kept in 32 bits: the tensor core's sums lose with the length of the chain, and one accumulator over all of K was further off 64 bits than the
  // pieces that the streaming kernel cuts (K of 22528: 2.6e-5 of the norm against 1.9e-5, 4096: 4.4e-6 / 3.9e-6). Each half of K has an accumulator of
  // its own, added at the end; the next tile then waits for the epilogue. Outputs in bf16 round away 1.7e-3.
  s.halves = p.mode == 0 && p.out_f32 && s.KB >= 32;
}

// A pair's work: its piece of a cut tile, then whole tiles R + c, R + c + pairs, ...
struct PairWalk {
  int piece, next;
  bool cut = false, more = false;      // of the step just taken: a piece of a cut tile; a first half, whose second one comes next
  __device__ __forceinline__ PairWalk(const PairSched& s, int c) : piece(c < s.R * s.split ? c : -1), next(s.R + c) {}
  __device__ __forceinline__ bool step(const PairSched& s, int pairs, int& u, int& kb0, int& kb1) {
    if (piece >= 0) {
      // neighbouring pairs take the same K range of neighbouring tiles
      const int i = piece / s.R;
      u = piece - i * s.R;
      kb0 = i * s.KB / s.split;
      kb1 = (i + 1) * s.KB / s.split;
      piece = -1;
      cut = true;
      return true;
    }
    cut = false;
    if (next >= s.U) return false;
    u = next;
    more = s.halves && !more;      // (false before the first step)
    kb0 = s.halves && !more ? s.KB / 2 : 0;
    kb1 = more ? s.KB / 2 : s.KB;
    if (!more) next += pairs;
    return true;
  }
};

__device__ __forceinline__ Unit pair_unit(const PairSched& s, int G, int u) {
  int g = 0;
  while (g + 1 < G && u >= s.pre[g + 1]) ++g;
  const int r = u - s.pre[g], nt = s.ntile[g], band = r / (RASTER * nt), rb = r - band * RASTER * nt, bm = min(s.MT - band * RASTER, RASTER);
  Unit x;
  x.g = g;
  x.n = rb / bm;
  x.m = band * RASTER + rb - x.n * bm;
  return x;
}

// ---- cluster and cta_group::2 forms ----
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// into this CTA's shared memory, completing on a barrier of the pair's even CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {      // arrives on both CTAs' barriers
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

template <bool DUAL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const PairArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ PairSched sched;
  __shared__ __align__(8) uint64_t bar_full[PAIR_STAGES], bar_empty[PAIR_STAGES], bar_tfull[2], bar_tempty[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag, all_here;

  const SkeinGemmParams& p = a.p;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int stage_bytes = PAIR_W_BYTES + a.x_box * 128;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_tfull[b]), 1);
      mbar_init(smem_u32(&bar_tempty[b]), 8);       // the epilogue warps of both CTAs
    }
    fence_mbar_init();
    pair_sched(sched, p, a.cap, pairs);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base_smem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && elect_one()) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();       // both CTAs' barriers are set up before either is signalled
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  const int KB = sched.KB;

  if (warp == 0) {
    // ================= TMA producer =================
    if (elect_one()) {
      PairWalk walk(sched, pair);
      uint32_t it = 0;
      int u, kb0, kb1;
      bool ok = true;
      while (ok && walk.step(sched, pairs, u, kb0, kb1)) {
        const Unit un = pair_unit(sched, p.G, u);
        const int w_row = un.g * p.w_rows_per_group + (DUAL ? un.m * 128 + (int)rank * 64 : un.m * 256 + (int)rank * 128);
        const int cols = sched.cols[un.g];
        const int x_row = sched.off[un.g] + un.n * cols + (int)rank * (cols >> 1);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % a.stages, ph = (it / a.stages) & 1;
          if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1, &abort_flag, a.budget_ns)) {
            report_status(p.status, ST_TIMEOUT_SMEM_EMPTY, blockIdx.x);
            abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t full = map_to_rank(smem_u32(&bar_full[s]), 0);
          const uint32_t st = smem_base + s * stage_bytes;
          if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2u * stage_bytes);      // the copies of both CTAs
          if (DUAL) {
            const int up = w_row + p.up_row_off;
            if (p.w_packed) {
              tma_load_2d_pair(st, &tmW, full, 0, ((w_row >> 7) * KB + kb) * 128 + (w_row & 127));
              tma_load_2d_pair(st + PAIR_W_BYTES / 2, &tmW, full, 0, ((up >> 7) * KB + kb) * 128 + (up & 127));
            } else {
              tma_load_2d_pair(st, &tmW, full, kb * 64, w_row);
              tma_load_2d_pair(st + PAIR_W_BYTES / 2, &tmW, full, kb * 64, up);
            }
          } else if (p.w_packed) {
            tma_load_2d_pair(st, &tmW, full, 0, ((w_row >> 7) * KB + kb) * 128);
          } else {
            tma_load_2d_pair(st, &tmW, full, kb * 64, w_row);
          }
          tma_load_2d_pair(st + PAIR_W_BYTES, &tmX, full, kb * 64, x_row);
        }
      }
      // The MMA's commits arrive on both CTAs' barriers: nobody leaves before the last one on every stage is here (a stage never filled passes).
      for (int i = 0; ok && i < a.stages; ++i, ++it) {
        const uint32_t s = it % a.stages;
        if (!mbar_wait(smem_u32(&bar_empty[s]), ((it / a.stages) & 1) ^ 1, &abort_flag, a.budget_ns)) {
          report_status(p.status, ST_TIMEOUT_SMEM_EMPTY, blockIdx.x);
          abort_flag = 1;
          ok = false;
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer of the pair =================
    if (rank == 0 && elect_one()) {
      PairWalk walk(sched, pair);
      uint32_t it = 0, seg = 0;
      int u, kb0, kb1;
      bool ok = true;
      for (; ok && walk.step(sched, pairs, u, kb0, kb1); ++seg) {
        const Unit un = pair_unit(sched, p.G, u);
        const uint32_t idesc = umma_idesc(1, 1, 256, sched.cols[un.g]);
        const uint32_t b = seg & 1;
        if (!mbar_wait(smem_u32(&bar_tempty[b]), ((seg >> 1) & 1) ^ 1, &abort_flag, a.budget_ns)) {
          report_status(p.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x);
          abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + b * PAIR_COLS;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % a.stages;
          if (!mbar_wait(smem_u32(&bar_full[s]), (it / a.stages) & 1, &abort_flag, a.budget_ns)) {
            report_status(p.status, ST_TIMEOUT_SMEM_FULL, blockIdx.x);
            abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t st = smem_base + s * stage_bytes;
          const uint64_t dw = umma_desc_sw128(st), dx = umma_desc_sw128(st + PAIR_W_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_pair(d_tmem, dw + 2 * k, dx + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          tc_commit_pair(smem_u32(&bar_empty[s]));
        }
        if (ok) tc_commit_pair(smem_u32(&bar_tfull[b]));
      }
    }
  } else {
    // ================= epilogue (warps 2..5) =================
    const int q = warp & 3, r = q * 32 + lane, et = threadIdx.x - 64;
    const size_t slot_elems = (size_t)PAIR_ROWS * PAIR_COLS;
    float* xch = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)) + a.stages * stage_bytes);
    const uint32_t leader_tempty[2] = {map_to_rank(smem_u32(&bar_tempty[0]), 0), map_to_rank(smem_u32(&bar_tempty[1]), 0)};
    const bool pairs_ok = !p.out_f32 && p.ldo % 2 == 0 && p.out_col0 % 2 == 0 && (((uintptr_t)p.out | (uintptr_t)p.residual) & 3) == 0 && p.F % 2 == 0;
    const bool quads_ok = p.out_f32 && p.ldo % 4 == 0 && p.out_col0 % 4 == 0 && (((uintptr_t)p.out | (uintptr_t)p.residual) & 15) == 0 && p.F % 4 == 0;
    const int odd = lane & 1;
    // one output, wherever it comes from
    auto emit = [&](float y, long long row, int f) {
      const size_t idx = (size_t)row * p.ldo + p.out_col0 + f;
      if (f < p.relu2_cols) y = relu2(y);
      if (p.out_f32) { ((float*)p.out)[idx] = p.residual ? y + ((const float*)p.residual)[idx] : y; return; }
      if (p.residual) y += __bfloat162float(((const __nv_bfloat16*)p.residual)[idx]);
      ((__nv_bfloat16*)p.out)[idx] = __float2bfloat16(y);
    };
    // bf16 rows: neighbouring lanes (features) exchange, so that a lane stores two features of every other token. res: the residuals there, or null
    auto store_pairs = [&](const float* y, int n, long long row, int left, int f, const __nv_bfloat162* res) {   // left: tokens from `row` on
      __nv_bfloat16* out = (__nv_bfloat16*)p.out + (size_t)(row + odd) * p.ldo + p.out_col0 + f - odd;
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        if (j >= n) break;
        const float got = __shfl_xor_sync(0xffffffffu, odd ? y[j] : y[j + 1], 1), own = odd ? y[j + 1] : y[j];
        float2 v = odd ? make_float2(got, own) : make_float2(own, got);
        if (res) { const float2 r2 = __bfloat1622float2(res[j / 2]); v.x += r2.x; v.y += r2.y; }
        if (f < p.F && j + odd < left) *reinterpret_cast<__nv_bfloat162*>(out + (size_t)j * p.ldo) = __floats2bfloat162_rn(v.x, v.y);
      }
    };
    // sum of the tile that this pair has a piece of: this CTA's run of token columns, pieces in order
    int parked = -1;
    bool ok = true;
    auto reduce_parked = [&]() {
      const Unit un = pair_unit(sched, p.G, parked);
      const int nc = sched.split, mine = (pair - parked) / sched.R;
      int* counter = &p.counters[parked * 2 + (int)rank];
      if (et == 0) {
        int here = 0;
        const uint64_t t0 = global_timer_ns();
        for (;;) {
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(here) : "l"(counter) : "memory");
          here &= 0xffff;
          if (here >= nc || *(volatile int*)&abort_flag || global_timer_ns() - t0 > a.budget_ns) break;
        }
        if (here < nc) {
          report_status(p.status, ST_TIMEOUT_SPLITK, blockIdx.x);
          abort_flag = 1;
        }
        all_here = here >= nc;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (!all_here) { ok = false; return; }
      const int cols = sched.cols[un.g];
      const int valid = min(cols, sched.cnt[un.g] - un.n * cols);
      const long long row0 = (long long)sched.off[un.g] + (long long)un.n * cols;
      const int c_lo = (int)((long long)valid * mine / nc), c_hi = (int)((long long)valid * (mine + 1) / nc);
      // a thread sums 4 consecutive features of CB columns: a warp's load is one column (a gate/up pair: two), CB of them per contributor
      // in flight
      constexpr int FL = DUAL ? 16 : 32, CB = DUAL ? 4 : 8;
      const int fl = (lane % FL) * 4, f = (DUAL ? un.m * 128 + (int)rank * 64 : un.m * 256 + (int)rank * 128) + fl;
      const int step = 4 * (32 / FL);                       // columns that the four warps load at once
      for (int c0 = c_lo + (warp - 2) * (32 / FL) + lane / FL; c0 < c_hi; c0 += step * CB) {
        float4 y[CB], z[CB];
        float4 rv[CB];                                        // residuals, ahead of the partials
        if ((pairs_ok || quads_ok) && p.residual != nullptr) {
#pragma unroll
          for (int j = 0; j < CB; ++j) {
            const size_t at = (size_t)(row0 + min(c0 + j * step, c_hi - 1)) * p.ldo + p.out_col0 + f;
            if (quads_ok) {
              if (f < p.F) rv[j] = *reinterpret_cast<const float4*>((const float*)p.residual + at);
            } else {
              const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>((const __nv_bfloat16*)p.residual + at);
              const float2 a0 = f < p.F ? __bfloat1622float2(r2[0]) : make_float2(0.f, 0.f), a1 = f + 2 < p.F ? __bfloat1622float2(r2[1]) : make_float2(0.f, 0.f);
              rv[j] = make_float4(a0.x, a0.y, a1.x, a1.y);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < CB; ++j) y[j] = z[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = 0; i < nc; ++i) {
          const float* ws = p.workspace + (size_t)(2 * (i * sched.R + parked) + (int)rank) * slot_elems + fl;
          float4 v[CB], w[CB];
#pragma unroll
          for (int j = 0; j < CB; ++j) {
            const float* at = ws + (size_t)min(c0 + j * step, c_hi - 1) * PAIR_ROWS;
            v[j] = __ldcg(reinterpret_cast<const float4*>(at));
            if (DUAL) w[j] = __ldcg(reinterpret_cast<const float4*>(at + 64));
          }
#pragma unroll
          for (int j = 0; j < CB; ++j) {
            y[j].x += v[j].x; y[j].y += v[j].y; y[j].z += v[j].z; y[j].w += v[j].w;
            if (DUAL) { z[j].x += w[j].x; z[j].y += w[j].y; z[j].z += w[j].z; z[j].w += w[j].w; }
          }
        }
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          const int col = c0 + j * step;
          if (col >= c_hi) break;
          float o[4] = {y[j].x, y[j].y, y[j].z, y[j].w};
          if (DUAL) {
            o[0] = glu_act(p, o[0], z[j].x); o[1] = glu_act(p, o[1], z[j].y); o[2] = glu_act(p, o[2], z[j].z); o[3] = glu_act(p, o[3], z[j].w);
          }
          if (pairs_ok || quads_ok) {
            const size_t first = (size_t)(row0 + col) * p.ldo + p.out_col0 + f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (f + i < p.relu2_cols) o[i] = relu2(o[i]);
            if (p.residual != nullptr) { o[0] += rv[j].x; o[1] += rv[j].y; o[2] += rv[j].z; o[3] += rv[j].w; }
            if (quads_ok) {
              if (f < p.F) *reinterpret_cast<float4*>((float*)p.out + first) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
#pragma unroll
              for (int i = 0; i < 4; i += 2)
                if (f + i < p.F) *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)p.out + first + i) = __floats2bfloat162_rn(o[i], o[i + 1]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (f + i < p.F) emit(o[i], row0 + col, f + i);
          }
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (et == 0) {
        const int old = atomicAdd(counter, 0x10000);
        if ((old >> 16) == nc - 1) *counter = 0;       // the last one out re-arms it for the next launch
      }
      parked = -1;
    };

    PairWalk walk(sched, pair);
    uint32_t seg = 0;
    int u, kb0, kb1, buf = 0;
    for (; ok && walk.step(sched, pairs, u, kb0, kb1); ++seg) {
      if (parked >= 0) {
        reduce_parked();
        if (!ok) break;
      }
      const Unit un = pair_unit(sched, p.G, u);
      const uint32_t b = seg & 1;
      if (!mbar_wait(smem_u32(&bar_tfull[b]), (seg >> 1) & 1, &abort_flag, a.budget_ns)) {
        report_status(p.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x);
        abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      if (walk.more) continue;               // the first half stays in its accumulator until the second one is there
      const bool halves = sched.halves && !walk.cut;
      const uint32_t t_acc = tmem_base + b * PAIR_COLS + ((uint32_t)(q * 32) << 16), t_first = tmem_base + (b ^ 1) * PAIR_COLS + ((uint32_t)(q * 32) << 16);
      const int cols = sched.cols[un.g];
      const int valid = min(cols, sched.cnt[un.g] - un.n * cols);
      const long long row0 = (long long)sched.off[un.g] + (long long)un.n * cols;
      if (walk.cut) {
        float* ws = p.workspace + (size_t)blockIdx.x * slot_elems;
        for (int c0 = 0; c0 < valid; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(t_acc + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) __stcg(ws + (size_t)(c0 + j) * PAIR_ROWS + r, __uint_as_float(v[j]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_tempty[b]);
        asm volatile("bar.sync 1, 128;" ::: "memory");      // the 128 threads' partials before the release that publishes them
        if (et == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&p.counters[u * 2 + (int)rank]) : "memory");
        parked = u;
        continue;
      }
      for (int c0 = 0; c0 < valid; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(t_acc + c0, v);
        if (DUAL) {
          // lanes 0-63 hold gates, 64-127 the matching ups: a gate warp gives the second 16 columns away and finishes the first 16, its up
          // warp the other way round
          const int f = un.m * 128 + (int)rank * 64 + (q & 1) * 32 + lane;
          const bool up = q >= 2;
          float* mine = xch + (((buf * 2 + (q & 1)) * 2 + (up ? 1 : 0)) * 16) * 32 + lane;
          const float* theirs = xch + (((buf * 2 + (q & 1)) * 2 + (up ? 0 : 1)) * 16) * 32 + lane;
          buf ^= 1;
          tmem_ld_wait();
          float y[32];
#pragma unroll
          for (int j = 0; j < 16; ++j) mine[j * 32] = __uint_as_float(up ? v[j] : v[16 + j]);
          asm volatile("bar.sync %0, 64;" ::"r"(2 + (q & 1)) : "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float o = theirs[j * 32], w = __uint_as_float(up ? v[16 + j] : v[j]);
            y[j] = glu_act(p, up ? o : w, up ? w : o);
          }
          const int c1 = c0 + (up ? 16 : 0);
          if (pairs_ok && p.residual == nullptr && p.relu2_cols == 0) {
            store_pairs(y, 16, row0 + c1, valid - c1, f, nullptr);
          } else if (f < p.F) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (c1 + j < valid) emit(y[j], row0 + c1 + j, f);
          }
        } else {
          const int f = un.m * 256 + (int)rank * 128 + r;
          // Residuals, usually in place: those of the 32 columns are on their way before the first sum is stored (one at a time, a load waited for the
          // store before: 3000 rows of 4096 x 4096 with bf16 residuals 418 us).
          if (p.out_f32) {
            const size_t first = (size_t)row0 * p.ldo + p.out_col0 + f;
            float rv[32];
            if (p.residual != nullptr && f < p.F) {
              const float* res = (const float*)p.residual + first;
#pragma unroll
              for (int j = 0; j < 32; ++j) rv[j] = __ldcg(res + (size_t)min(c0 + j, valid - 1) * p.ldo);
            }
            uint32_t v1[32];
            if (halves) tmem_ld32(t_first + c0, v1);
            tmem_ld_wait();
            if (f < p.F) {
              float* out = (float*)p.out + first;
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                float y = __uint_as_float(v[j]);
                if (halves) y += __uint_as_float(v1[j]);
                if (f < p.relu2_cols) y = relu2(y);
                if (p.residual != nullptr) y += rv[j];
                if (c0 + j < valid) out[(size_t)(c0 + j) * p.ldo] = y;
              }
            }
          } else {
            __nv_bfloat162 rp[16];
            if (pairs_ok && p.residual != nullptr && f < p.F) {
              const __nv_bfloat16* res = (const __nv_bfloat16*)p.residual + (size_t)row0 * p.ldo + p.out_col0 + f - odd;
#pragma unroll
              for (int j = 0; j < 32; j += 2)
                rp[j / 2] = *reinterpret_cast<const __nv_bfloat162*>(res + (size_t)min(c0 + j + odd, valid - 1) * p.ldo);
            }
            tmem_ld_wait();
            float y[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(v[j]);
            if (pairs_ok) {
              if (f < p.relu2_cols) {
#pragma unroll
                for (int j = 0; j < 32; ++j) y[j] = relu2(y[j]);
              }
              store_pairs(y, 32, row0 + c0, valid - c0, f, p.residual != nullptr ? rp : nullptr);
            } else if (f < p.F) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (c0 + j < valid) emit(y[j], row0 + c0 + j, f);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (halves) mbar_arrive_cluster(leader_tempty[b ^ 1]);
        mbar_arrive_cluster(leader_tempty[b]);
      }
    }
    if (ok && parked >= 0) reduce_parked();
  }

  // ---- tear-down: nobody leaves while the peer may still signal or read this CTA's shared memory ----
  if (*(volatile int*)&abort_flag) {
    // copies and MMAs that are still in flight land before the memory is given back
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// CTAs that fit at once, or a negative error: the cut tiles' sums need all of them resident.
template <bool DUAL>
static int pair_grid() {
  static PerDevice grid;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -7;
  return grid.get(dev, [] {
    if (cudaFuncSetAttribute(gemm_pair_kernel<DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM_MAX) != cudaSuccess) return -7;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(skein_sm_count() & ~1);
    cfg.blockDim = dim3(PAIR_THREADS);
    cfg.dynamicSmemBytes = PAIR_SMEM_MAX;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2; at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<DUAL>, &cfg) != cudaSuccess || n < 1) return -7;
    n = n * 2 < skein_sm_count() ? n * 2 : skein_sm_count() & ~1;
    return n < 148 ? n : 148;       // the workspace and the counters hold this many CTAs' partials
  });
}

// Tokens of a tile for `rows` rows: the width for which the rounds of whole and cut tiles cost least, where a K-block of a tile costs the
// bytes that it stages (128 weight rows and half of its tokens per CTA). Narrower than 256 pays where that fills a round: 512 rows of 6144
// features are 72 tiles of 192 instead of 48 of 256 (see the sizes at pair_gemm_ok in ops/functional.py).
static int pair_cap(int rows, int MT, int KB, int pairs) {
  long long best = 0;
  int cap = PAIR_COLS;
  for (int nt = pair_tiles(rows, PAIR_COLS), i = 0; i < 8; ++i, ++nt) {
    const int cols = ((rows + nt - 1) / nt + 31) / 32 * 32, tiles = pair_tiles(rows, cols);
    const long long U = (long long)MT * tiles;
    const int R = (int)(U % pairs), sp = pair_split(R, KB, pairs);
    const long long kbs = U / pairs * KB + (R == 0 ? 0 : sp > 1 ? (KB + sp - 1) / sp + 12 : KB), cost = kbs * (128 + cols / 2);
    if (i == 0 || cost < best) { best = cost; cap = cols; }
  }
  return cap;
}

}  // namespace skein

// The same contract as skein_gemm_ws (gemm_ws.cuh) for bf16 operands without publish, output gate or per-head columns; n_tile, stages, grid
// and line_cut_only are not read. Returns 0, a cudaError_t or a negative argument-error code.
extern "C" int skein_gemm_pair(const SkeinGemmParams* p, void* stream) {
  using namespace skein;
  if (!p || p->G < 1 || p->G > SKEIN_MAX_GROUPS) return -1;
  if (p->K <= 0 || p->K % (p->w_packed ? 64 : 8) != 0 || p->F <= 0) return -2;
  if (p->x_ld % 8 != 0 || (p->x_ld != 0 && p->x_ld < p->K)) return -2;
  if (p->mode < 0 || p->mode > 1 || p->fp8 != 0 || p->gate != nullptr || p->x_group_cols != 0 || p->out_group_cols != 0) return -4;
  if (!p->workspace || !p->counters) return -8;
  const bool dual = p->mode == 1;
  if (p->w_packed && (p->w_rows_per_group % 128 != 0 || (dual && p->up_row_off % 128 != 0))) return -9;
  const int grid = dual ? pair_grid<true>() : pair_grid<false>();
  if (grid < 0) return grid;
  PairArgs a;
  a.p = *p;
  const int ft = dual ? PAIR_ROWS : 2 * PAIR_ROWS;
  a.cap = p->group_cnt ? PAIR_COLS : pair_cap(p->t_static, (p->F + ft - 1) / ft, (p->K + 63) / 64, grid / 2);
  a.x_box = (p->group_cnt ? PAIR_COLS : pair_cols(p->t_static, a.cap)) / 2;
  const int stage = PAIR_W_BYTES + a.x_box * 128, xch = dual ? PAIR_XCH_FLOATS * 4 : 0;
  a.stages = (PAIR_SMEM_MAX - 1024 - xch) / stage;
  if (a.stages > PAIR_STAGES) a.stages = PAIR_STAGES;
  a.budget_ns = (uint64_t)(p->wait_budget_ms > 0 ? p->wait_budget_ms : gemm_wait_budget_ms()) * 1000000ull;
  CUtensorMap tmW, tmX;
  const uint64_t rows = (uint64_t)p->G * p->w_rows_per_group;
  const uint32_t w_box = dual ? 64 : 128;
  int rc = p->w_packed ? cached_tmap_2d(&tmW, p->W, rows * (p->K / 64), 64, 2, w_box) : cached_tmap_2d(&tmW, p->W, rows, p->K, 2, w_box);
  if (rc) return rc;
  rc = cached_tmap_2d_ld(&tmX, p->X, p->x_rows, p->K, p->x_ld > 0 ? p->x_ld : p->K, 2, a.x_box);
  if (rc) return rc;
  const size_t smem = (size_t)a.stages * stage + xch + 1024;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dual) gemm_pair_kernel<true><<<grid, PAIR_THREADS, smem, s>>>(tmW, tmX, a);
  else gemm_pair_kernel<false><<<grid, PAIR_THREADS, smem, s>>>(tmW, tmX, a);
  return (int)cudaGetLastError();
}
