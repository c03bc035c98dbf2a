// Causal prefill attention over the paged KV cache on the 5th-generation tensor cores (tcgen05, accumulators in
// tensor memory, operands staged by TMA). Same contract as attn_prefill.cu (chunked-prefill aware: a chunk of q_len
// new tokens attends to the kv_len tokens already in the cache, its own included); this is the kernel the prefill
// path runs for head sizes 128 and 64 and pages of whole 16-token groups, the mma.sync kernel stays as the fallback for other
// shapes. With a window or chunks (SkeinAttnRule) a row sees part of the keys before it only; tiles before the first key of a CTA's first
// row are skipped, but for those of the first tokens that the window keeps in sight.
//
// Differential heads (two maps over the same values, side by side in the 128 columns of a query or key head): the tile's 128 rows are two
// maps of 64 query rows, each with the other map's half set to zero, so that one product gives both maps' scores; at the end the rows of
// the second map hand their outputs over through shared memory, and the rows of the first one subtract, norm and gate them.
//
// Heads of one map take attn_prefill_pair_kernel (below), two heads of a group per CTA. With two maps one CTA has 64 query rows of one head, walking the
// context in 128-token tiles:
//
//   warp 0      TMA producer: the Q tile once, then per context tile the K pages and the V pages of the tile
//               (one 16-token x 64-element box per page and head-dim half, 128-byte swizzle) into single K and V
//               buffers; a lane per box, its page looked up a tile ahead
//   warp 1      MMA issuer (one elected lane): S = Q K^T (M 128 queries, N 128 tokens, K = head dim, both operands
//               K-major in shared memory, accumulator S in tensor memory), and O += P V with P taken from TENSOR
//               MEMORY as the A operand and the V tile as an MN-major B operand (tokens are the reduction dimension
//               and the cache stores a token's 128 values contiguously), accumulator O in tensor memory
//   warps 2-5   softmax: thread t owns query row t (tensor-memory lane t). Two passes over the row of S (row max,
//               then exp2 / row sum / bf16 P written back over the first half of S's columns); O is rescaled in
//               tensor memory only when some row of the warp raised its maximum; the last tile's rows are normalised
//               and stored from registers
//
// S (128 columns), P (aliased on S) and O (128 columns) take 256 tensor-memory columns and the three operand buffers
// 96 KB of shared memory, so TWO CTAs are resident per SM: while one CTA's softmax warps work on a tile, the other
// CTA's MMAs use the tensor cores. Every wait is bounded; on expiry the CTA records a status code, waits (bounded) for
// its copies in flight, frees its tensor memory and returns.
//
// The reference never runs a prefill attention kernel: its FlashInfer prefill wrapper returns -1
// (vendor/luminal/crates/luminal_cuda_lite/src/host/flashinfer/wrapper.cu:263-281) and prefill falls back to unfused
// graph ops (crates/skein_emit/src/op_wiring.rs:2155-2305).
#include "attn_rule.cuh"
#include "ptx.cuh"
#include "launch.cuh"
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>

namespace skein {

int cached_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t k_elems, int elem_bytes, uint32_t box_rows);

constexpr int TC_BM = 128, TC_BN = 128, TC_PS = 16;    // (TC_PS: tokens of one box; a page is a multiple of it)
constexpr int TC_THREADS = 192;
constexpr int TC_HALF_BYTES = 128 * 128;              // one 64-element half of a 128-row tile, 128-byte rows
constexpr int TC_TMEM_COLS = 256;
constexpr uint64_t TC_BUDGET_NS = 4000000000ull;

struct AttnPrefillTcParams {
  const int* block_table;   // [S, max_blocks]
  const int* q_start;       // [S] first row of the sequence's chunk in q / out
  const int* q_len;         // [S]
  const int* kv_len;        // [S] tokens in the cache after this chunk was appended
  __nv_bfloat16* out;       // [T, Hq * D]
  int* status;
  int Hq, Hkv, max_blocks, num_pages, page_size;
  long long out_ld;         // elements between rows of out
  float scale_log2e, cap_in, cap_log2e;      // (cap_log2e 0: scores are not capped; attn_cap)
  SkeinAttnRule r;
};

constexpr int TC_X_LD = 132;            // floats between rows of the second map's outputs in shared memory

__global__ void __launch_bounds__(TC_THREADS, 2)
attn_prefill_maps_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                       const AttnPrefillTcParams p) {
  constexpr int TC_D = 128, HALVES = 2, TC_TILE_BYTES = HALVES * TC_HALF_BYTES;      // two maps fill the two halves of a head
  constexpr int QR = TC_BM / 2;                             // query rows of a tile
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;     // long rows first: the causal work grows with the row
  const int head = blockIdx.y, seq = blockIdx.z;
  const int qlen = p.q_len[seq];
  const int q0 = qt * QR;
  if (q0 >= qlen) return;
  const int kvlen = p.kv_len[seq];
  const int pos0 = kvlen - qlen;                            // absolute position of the chunk's first token
  const int qrow0 = p.q_start[seq];
  const int kvh = head / (p.Hq / p.Hkv);
  int kv_hi = pos0 + min(q0 + QR, qlen);                    // exclusive bound of the keys any row of this tile sees
  if (kv_hi > kvlen) kv_hi = kvlen;
  const int kv_lo = attn_first_key(p.r.window, p.r.chunk, pos0 + q0);                    // first key of the first row
  const int last_lo = attn_first_key(p.r.window, p.r.chunk, pos0 + q0 + QR - 1);         // ... and of the last
  const int keep = p.r.keep_first;
  const int first_tile = kv_lo / TC_BN;
  const int kept = min((keep + TC_BN - 1) / TC_BN, first_tile);                          // tiles of the kept first tokens ...
  const int n_tiles = (kv_hi + TC_BN - 1) / TC_BN - first_tile + kept;                   // ... in front of the window's
  auto tile_at = [&](int j) { return j < kept ? j : first_tile + j - kept; };
  // tokens of tile j that some row sees, counted from its first
  auto tile_len = [&](int j) { return min(j < kept ? keep : kv_hi, (tile_at(j) + 1) * TC_BN) - tile_at(j) * TC_BN; };

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_s = base, k_s = base + TC_TILE_BYTES, v_s = base + 2 * TC_TILE_BYTES;
  const uint32_t bars = base + 3 * TC_TILE_BYTES;
  const uint32_t bar_q = bars, bar_kfull = bars + 8, bar_kempty = bars + 16, bar_vfull = bars + 24, bar_vempty = bars + 32,
                 bar_sfull = bars + 40, bar_pfull = bars + 48, bar_odone = bars + 56;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + 3 * TC_TILE_BYTES + 64);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + 3 * TC_TILE_BYTES + 72);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(bar_q, 1); mbar_init(bar_kfull, 1); mbar_init(bar_kempty, 1); mbar_init(bar_vfull, 1);
    mbar_init(bar_vempty, 1); mbar_init(bar_sfull, 1); mbar_init(bar_pfull, 128); mbar_init(bar_odone, 1);
    abort_flag[0] = 0;
    abort_flag[1] = 0;      // never set: the drain waits of a failing producer run out on their time budget only
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TC_TMEM_COLS);
    tmem_relinquish();
  }
  for (int i = tid; i < 2 * 64 * 8; i += TC_THREADS) {      // the halves of Q that no copy fills: rows 64 .. of the first, rows .. 63 of the second
    const uint32_t a = q_s + (i < 64 * 8 ? 64 * 128 + i * 16 : TC_HALF_BYTES + (i - 64 * 8) * 16);
    asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(a), "r"(0) : "memory");
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_s = tmem, tm_p = tmem, tm_o = tmem + 128;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    const uint64_t pol_q = l2_policy_evict_first(), pol_kv = l2_policy_evict_last();
    if (lane == 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmKV);
      mbar_expect_tx(bar_q, TC_TILE_BYTES / 2);
      for (int hf = 0; hf < HALVES; ++hf)
        tma_load_2d(q_s + hf * TC_HALF_BYTES + hf * 64 * 128, &tmQ, bar_q, head * TC_D + hf * 64, qrow0 + q0, pol_q);
    }
    const int* bt = p.block_table + (size_t)seq * p.max_blocks;
    auto page_of = [&](int j) {
      const int tok = tile_at(j) * TC_BN + lane * TC_PS;
      return j < n_tiles && lane * TC_PS < tile_len(j) ? bt[tok / p.page_size] : 0;
    };
    bool ok = true;
    int armed_k = 0, armed_v = 0;      // phases armed so far (for the bounded drain on an early exit)
    for (int j = 0, next = page_of(0); j < n_tiles && ok; ++j) {
      const int n_pages = (tile_len(j) + TC_PS - 1) / TC_PS, in_page = (tile_at(j) * TC_BN + lane * TC_PS) % p.page_size;
      int page = next;
      next = page_of(j + 1);
      if (page < 0 || page >= p.num_pages) { report_status(p.status, ST_BAD_INDEX, page); page = 0; }
      for (int kv01 = 0; kv01 < 2; ++kv01) {
        const uint32_t full = kv01 ? bar_vfull : bar_kfull, empty = kv01 ? bar_vempty : bar_kempty;
        const uint32_t dst = (kv01 ? v_s : k_s) + lane * TC_PS * 128;
        ok = __all_sync(0xffffffffu, j == 0 || mbar_wait(empty, (j - 1) & 1, abort_flag, TC_BUDGET_NS));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(full, (uint32_t)n_pages * HALVES * TC_PS * 128);
        if (kv01) ++armed_v; else ++armed_k;
        __syncwarp();
        if (lane < n_pages) {
          const int row = ((page * 2 + kv01) * p.Hkv + kvh) * p.page_size + in_page;
          for (int hf = 0; hf < HALVES; ++hf) tma_load_2d(dst + hf * TC_HALF_BYTES, &tmKV, full, hf * 64, row, pol_kv);
        }
      }
    }
    if (!ok && lane == 0) {
      if (*abort_flag == 0) { *abort_flag = 1; report_status(p.status, ST_TIMEOUT_SMEM_EMPTY, 10); }
      // copies already issued still write this CTA's shared memory: wait for them (bounded) before leaving
      if (armed_k > 0) mbar_wait(bar_kfull, (armed_k - 1) & 1, abort_flag + 1, TC_BUDGET_NS);
      if (armed_v > 0) mbar_wait(bar_vfull, (armed_v - 1) & 1, abort_flag + 1, TC_BUDGET_NS);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = umma_idesc(1, 1, TC_BM, TC_BN);
      const uint32_t idesc_o = umma_idesc(1, 1, TC_BM, TC_D) | (1u << 16);      // B operand MN-major
      bool ok = mbar_wait(bar_q, 0, abort_flag, TC_BUDGET_NS);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (!mbar_wait(bar_kfull, j & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < TC_D / 16; ++k) {
          const uint32_t off = (k >> 2) * TC_HALF_BYTES + (k & 3) * 32;
          mma_f16(tm_s, umma_desc_sw128(q_s + off), umma_desc_sw128(k_s + off), idesc_s, k > 0 ? 1u : 0u);
        }
        tc_commit(bar_kempty);
        tc_commit(bar_sfull);
        if (!mbar_wait(bar_pfull, j & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        if (!mbar_wait(bar_vfull, j & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        tc_fence_after();
        const int k_steps = (tile_len(j) + 15) / 16;               // 16-token steps that hold at least one visible key
        for (int k = 0; k < k_steps; ++k)
          mma_f16_ts(tm_o, tm_p + k * 8, umma_desc_sw128_mn(v_s + k * 16 * 128, TC_HALF_BYTES), idesc_o,
                     (j > 0 || k > 0) ? 1u : 0u);
        tc_commit(bar_vempty);
        tc_commit(bar_odone);
      }
      if (!ok && *abort_flag == 0) { *abort_flag = 1; report_status(p.status, ST_TIMEOUT_SMEM_FULL, 11); }
    }
  } else {
    // ---------------------------------------------------------------- softmax warps: thread <-> query row
    const int lane_grp = warp & 3;                      // the 32 tensor-memory lanes this warp may access
    const int r = lane_grp * 32 + lane;                 // row of the tile
    const uint32_t lane_addr = (uint32_t)(lane_grp * 32) << 16;
    const int qi = r % QR;                              // its query row (rows QR .. are the second map's)
    int pos_r = pos0 + q0 + qi;
    if (pos_r > kvlen - 1) pos_r = kvlen - 1;           // rows past the chunk are computed, finite, and never stored
    const int first_key = attn_first_key(p.r.window, p.r.chunk, pos_r);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const int n0 = tile_at(j) * TC_BN;
      if (!mbar_wait(bar_sfull, j & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
      tc_fence_after();
      // some row of the tile sees only part of these keys (the tile's last row has the latest window)
      const bool masked = n0 + TC_BN - 1 > pos0 + q0 || (n0 < last_lo && n0 + TC_BN > keep);
      const int limit = pos_r - n0;                     // this row sees columns first .. limit of the tile, and those before `until`
      const int first = first_key - n0, until = keep - n0;
      auto seen = [&](int c) { return c <= limit && (c >= first || c < until); };
      // pass 1: row maximum of the raw scores (64 columns per round: both loads in flight before the wait)
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int h = 0; h < TC_BN / 64; ++h) {
        uint32_t sv[64];
        tmem_ld32(tm_s + lane_addr + h * 64, sv);
        tmem_ld32(tm_s + lane_addr + h * 64 + 32, sv + 32);
        tmem_ld_wait();
        if (masked) {
#pragma unroll
          for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], seen(h * 64 + i) ? __uint_as_float(sv[i]) : -INFINITY);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
        }
      }
      const float raw = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));                   // the scale is positive, the cap monotonic
      const float mx = raw * p.scale_log2e;
      // The running maximum only moves when the tile's maximum exceeds it by more than 2^8: until then the
      // probabilities of this tile are at most 256 (exact in bf16 and harmless in the fp32 sums), and O needs no
      // rescaling; the final division by the row sum undoes whatever reference the row ended on.
      const float m_new = (m == -INFINITY || mx > m + 8.f) ? fmaxf(m, mx) : m;
      const float alpha = (m == -INFINITY) ? 1.f : exp2f(m - m_new);
      const float ref = m_new == -INFINITY ? 0.f : m_new;      // (a row whose window starts in a later tile)
      if (j > 0) {
        // O of the previous tiles is complete in tensor memory; bring it to the new reference if some row moved
        if (!mbar_wait(bar_odone, (j - 1) & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        tc_fence_after();
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
          for (int h = 0; h < TC_D / 64; ++h) {
            uint32_t ov[64];
            tmem_ld32(tm_o + lane_addr + h * 64, ov);
            tmem_ld32(tm_o + lane_addr + h * 64 + 32, ov + 32);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_st16(tm_o + lane_addr + h * 64 + c * 16, ov + c * 16);
          }
        }
      }
      l *= alpha;
      m = m_new;
      // pass 2: p = exp2(s * scale - m), row sum, bf16 pairs written over the columns of S already consumed
      float rs = 0.f;
#pragma unroll
      for (int h = 0; h < TC_BN / 64; ++h) {
        uint32_t sv[64];
        tmem_ld32(tm_s + lane_addr + h * 64, sv);
        tmem_ld32(tm_s + lane_addr + h * 64 + 32, sv + 32);
        tmem_ld_wait();
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          float x0 = fmaf(__uint_as_float(sv[i]), p.scale_log2e, -ref), x1 = fmaf(__uint_as_float(sv[i + 1]), p.scale_log2e, -ref);
          if (masked) {
            if (!seen(h * 64 + i)) x0 = -INFINITY;
            if (!seen(h * 64 + i + 1)) x1 = -INFINITY;
          }
          const float p0 = exp2f(x0), p1 = exp2f(x1);
          // the row sum is taken over the rounded values, the ones the tensor cores multiply
          const __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);
          const float2 pf = __bfloat1622float2(pb);
          rs += pf.x + pf.y;
          pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&pb);
        }
        // columns [32 h, 32 h + 32) of P lie inside columns [0, 64 h + 64) of S, all of which have been read
        tmem_st16(tm_p + lane_addr + h * 32, pk);
        tmem_st16(tm_p + lane_addr + h * 32 + 16, pk + 16);
      }
      l += rs;
      if (n0 + TC_BN > kv_hi) {
        // last tile: its final 16-token step may hold rows of V past the context (slots of the page that were never
        // written); zero them so that 0 * garbage cannot produce a NaN. Needs V landed; a 128-byte row is a
        // permutation of itself under the swizzle, so whole rows can be cleared without computing it.
        if (!mbar_wait(bar_vfull, j & 1, abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        const int past = kv_hi - n0;
        const int n_rows = ((past + 15) & ~15) - past;        // rows of the last 16-token step past the context
        for (int i = r; i < n_rows * 8; i += 128) {              // 16-byte chunks of those rows, per half
          const uint32_t a = v_s + past * 128 + i * 16;
#pragma unroll
          for (int hf = 0; hf < HALVES; ++hf)
            asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(a + hf * TC_HALF_BYTES), "r"(0) : "memory");
        }
        fence_proxy_async_smem();
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_pfull);
    }
    const bool done = ok && mbar_wait(bar_odone, (n_tiles - 1) & 1, abort_flag, TC_BUDGET_NS);
    const float inv = attn_norm(m, l, attn_sink_log2(p.r, head));
    const bool store = q0 + qi < qlen;
    // every copy and product of this CTA is complete: the K and V buffers take the second map's outputs
    float* x_row = reinterpret_cast<float*>(base_ptr + TC_TILE_BYTES) + (size_t)qi * TC_X_LD;
    if (done && r >= QR) {
      tc_fence_after();
      const float f = inv * p.r.lam[0];
#pragma unroll
      for (int c = 0; c < TC_D / 16; ++c) {
        uint32_t ov[16];
        tmem_ld16(tm_o + lane_addr + c * 16, ov);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<float4*>(x_row + c * 16 + i) = make_float4(__uint_as_float(ov[i]) * f, __uint_as_float(ov[i + 1]) * f,
                                                                       __uint_as_float(ov[i + 2]) * f, __uint_as_float(ov[i + 3]) * f);
      }
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");      // the four softmax warps, whatever their waits returned
    if (done && r < QR) {
      tc_fence_after();
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < TC_D / 16; ++c) {
        uint32_t ov[16];
        tmem_ld16(tm_o + lane_addr + c * 16, ov);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          float4 x = *reinterpret_cast<const float4*>(x_row + c * 16 + i);
          x.x = __uint_as_float(ov[i]) * inv - x.x; x.y = __uint_as_float(ov[i + 1]) * inv - x.y;
          x.z = __uint_as_float(ov[i + 2]) * inv - x.z; x.w = __uint_as_float(ov[i + 3]) * inv - x.w;
          ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
          *reinterpret_cast<float4*>(x_row + c * 16 + i) = x;
        }
      }
      const float f = p.r.out_scale / sqrtf(ss / (float)TC_D + p.r.eps);
      const size_t row = (size_t)(qrow0 + q0 + qi), col = (size_t)head * TC_D;
      if (store) {
        const __nv_bfloat16* g_row = p.r.gate ? (const __nv_bfloat16*)p.r.gate + row * p.r.gate_ld + col : nullptr;
#pragma unroll
        for (int c = 0; c < TC_D / 8; ++c) {
          float v[8];
          *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(x_row + c * 8);
          *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(x_row + c * 8 + 4);
          uint4 g4 = make_uint4(0, 0, 0, 0), o4;
          if (g_row) g4 = *reinterpret_cast<const uint4*>(g_row + c * 8);
          const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&g4);
          __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 a = make_float2(v[2 * i] * f, v[2 * i + 1] * f);
            if (g_row) {
              const float2 z = __bfloat1622float2(gb[i]);
              a.x /= 1.f + __expf(-z.x); a.y /= 1.f + __expf(-z.y);
            }
            ob[i] = __floats2bfloat162_rn(a.x, a.y);
          }
          *reinterpret_cast<uint4*>(p.out + row * p.out_ld + col + c * 8) = o4;
        }
      }
    }
    if (!done && *abort_flag == 0) {
      *abort_flag = 1;
      report_status(p.status, ST_TIMEOUT_TMEM_FULL, 12);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TC_TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// Heads of one map, two of a group at once. What bounds it is the chain of a tile: scores, row maximum, exponentials, values, of which the
// tensor cores take 1024 cycles of a 128 x 128 tile at head size 128 and the exponentials 1024 too (16 a cycle and SM). One CTA runs two such
// chains on one copy of the keys and values. Against a head per CTA and two CTAs per SM, each step behind the one before, a row of scores read
// twice and the block table read in front of every copy (which alone kept two chains waiting): 2048 rows behind 6144 cached, 32 heads 687 -> 262 us (350 -> 918 TFLOP/s), 8191
// rows, 64 heads 2922 -> 1082 us (1016), 8 x 512 rows, 32 heads 120 -> 53 us.
//
//   warps 0-3, 4-7   softmax of the first and of the second head: a thread holds its row's 128 scores in registers (one read of tensor memory)
//   warp 8           TMA producer: both Q tiles, then K and V tiles through a ring of four buffers, a lane per 16-token box, its page looked up a tile ahead
//   warp 9           MMA issuer: as soon as a head's probabilities are there, O += P V and the next tile's S = Q K^T back to back, so that one head's
//                    products run while the other's rows are in the softmax
//
// Tensor memory: S and P of the two heads in columns 0-127 and 128-255, their O behind: 512 columns, one CTA per SM. The commit after
// S(j + 1) follows O(j) on the same thread, so scores that have arrived say that O is complete up to the tile before.
// ---------------------------------------------------------------------------------------------
constexpr int TP_THREADS = 384, TP_SLOTS = 4;      // (the third warpgroup's last two warps only make it one)
constexpr int tp_smem(int d) { return (2 + TP_SLOTS) * (d / 64) * TC_HALF_BYTES + 1024 /* alignment slack */ + 256 /* barriers */; }

__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f32x2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f32x2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int TC_D, bool CAP>
__global__ void __launch_bounds__(TP_THREADS, 1)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, const AttnPrefillTcParams p) {
  constexpr int HALVES = TC_D / 64, TILE_BYTES = HALVES * TC_HALF_BYTES;
  const int group = p.Hq / p.Hkv, per_kv = (group + 1) / 2;
  const int kvh = blockIdx.x / per_kv, in_group = (blockIdx.x % per_kv) * 2, head0 = kvh * group + in_group;
  const int heads = min(2, group - in_group);               // an odd group's last head is alone
  const int seq = blockIdx.y;
  const int q0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * TC_BM;      // the last rows of all heads first: the causal work grows with the row
  const int qlen = p.q_len[seq];
  if (q0 >= qlen) return;
  const int kvlen = p.kv_len[seq], pos0 = kvlen - qlen, qrow0 = p.q_start[seq];
  const int kv_hi = min(kvlen, pos0 + min(q0 + TC_BM, qlen));         // as above: exclusive bound of the keys any row sees ...
  const int kv_lo = attn_first_key(p.r.window, p.r.chunk, pos0 + q0), last_lo = attn_first_key(p.r.window, p.r.chunk, pos0 + q0 + TC_BM - 1);
  const int keep = p.r.keep_first, first_tile = kv_lo / TC_BN;
  const int kept = min((keep + TC_BN - 1) / TC_BN, first_tile);
  const int n_tiles = (kv_hi + TC_BN - 1) / TC_BN - first_tile + kept;
  auto tile_at = [&](int j) { return j < kept ? j : first_tile + j - kept; };
  auto tile_len = [&](int j) { return min(j < kept ? keep : kv_hi, (tile_at(j) + 1) * TC_BN) - tile_at(j) * TC_BN; };

  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[TP_SLOTS], bar_empty[TP_SLOTS], bar_q, bar_s[2], bar_p[2], bar_o;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const uint32_t q_s = (smem_u32(smem_raw) + 1023u) & ~1023u, ring = q_s + 2 * TILE_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < TP_SLOTS; ++i) { mbar_init(smem_u32(&bar_full[i]), 1); mbar_init(smem_u32(&bar_empty[i]), 1); }
    for (int x = 0; x < 2; ++x) { mbar_init(smem_u32(&bar_s[x]), 1); mbar_init(smem_u32(&bar_p[x]), 4); }
    mbar_init(smem_u32(&bar_q), 1);
    mbar_init(smem_u32(&bar_o), 1);
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // 384 x 168 registers at launch = 2 x 128 x 208 + 128 x 88
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 8) {
      // ---------------------------------------------------------------- TMA producer
      const uint64_t pol_q = l2_policy_evict_first(), pol_kv = l2_policy_evict_last();
      if (lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmKV);
        mbar_expect_tx(smem_u32(&bar_q), heads * TILE_BYTES);
        for (int x = 0; x < heads; ++x)
          for (int hf = 0; hf < HALVES; ++hf)
            tma_load_2d(q_s + x * TILE_BYTES + hf * TC_HALF_BYTES, &tmQ, smem_u32(&bar_q), (head0 + x) * TC_D + hf * 64, qrow0 + q0, pol_q);
      }
      const int* bt = p.block_table + (size_t)seq * p.max_blocks;
      auto page_of = [&](int j) {
        const int tok = tile_at(j) * TC_BN + lane * TC_PS;
        return j < n_tiles && lane * TC_PS < tile_len(j) ? bt[tok / p.page_size] : 0;
      };
      bool ok = true;
      for (int j = 0, next = page_of(0); j < n_tiles && ok; ++j) {
        const int n_pages = (tile_len(j) + TC_PS - 1) / TC_PS, in_page = (tile_at(j) * TC_BN + lane * TC_PS) % p.page_size;
        int page = next;
        next = page_of(j + 1);
        if (page < 0 || page >= p.num_pages) { report_status(p.status, ST_BAD_INDEX, page); page = 0; }
        for (int kv01 = 0; kv01 < 2; ++kv01) {
          const int i = 2 * j + kv01, slot = i % TP_SLOTS;
          const uint32_t full = smem_u32(&bar_full[slot]), dst = ring + slot * TILE_BYTES + lane * TC_PS * 128;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[slot]), ((i / TP_SLOTS) & 1) ^ 1, &abort_flag, TC_BUDGET_NS));
          if (!ok) {
            if (lane == 0 && abort_flag == 0) report_status(p.status, ST_TIMEOUT_SMEM_EMPTY, 10);
            abort_flag = 1;
            break;
          }
          if (lane == 0) mbar_expect_tx(full, (uint32_t)n_pages * HALVES * TC_PS * 128);
          __syncwarp();
          if (lane < n_pages) {
            const int row = ((page * 2 + kv01) * p.Hkv + kvh) * p.page_size + in_page;
            for (int hf = 0; hf < HALVES; ++hf) tma_load_2d(dst + hf * TC_HALF_BYTES, &tmKV, full, hf * 64, row, pol_kv);
          }
        }
      }
    } else if (warp == 9) {
      // ---------------------------------------------------------------- MMA issuer
      if (lane == 0) {
        const uint32_t idesc_s = umma_idesc(1, 1, TC_BM, TC_BN);
        const uint32_t idesc_o = umma_idesc(1, 1, TC_BM, TC_D) | (1u << 16);      // B operand MN-major
        auto landed = [&](int i) { return mbar_wait(smem_u32(&bar_full[i % TP_SLOTS]), (i / TP_SLOTS) & 1, &abort_flag, TC_BUDGET_NS); };
        const uint64_t dq[2] = {umma_desc_sw128(q_s), umma_desc_sw128(q_s + TILE_BYTES)};
        const uint64_t dk = umma_desc_sw128(ring), dv = umma_desc_sw128_mn(ring, TC_HALF_BYTES);
        auto scores = [&](int x, int j) {
          const uint64_t a = dq[x], b = dk + (uint64_t)((2 * j % TP_SLOTS) * (TILE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < TC_D / 16; ++k) {
            const uint32_t off = ((k >> 2) * TC_HALF_BYTES + (k & 3) * 32) >> 4;
            mma_f16(tmem + x * 128, a + off, b + off, idesc_s, k > 0 ? 1u : 0u);
          }
          tc_commit(smem_u32(&bar_s[x]));
        };
        bool ok = mbar_wait(smem_u32(&bar_q), 0, &abort_flag, TC_BUDGET_NS) && landed(0);
        if (ok) {
          tc_fence_after();
          for (int x = 0; x < heads; ++x) scores(x, 0);
          tc_commit(smem_u32(&bar_empty[0]));
        }
        for (int j = 0; j < n_tiles && ok; ++j) {
          const bool more = j + 1 < n_tiles;
          if (more && !landed(2 * j + 2)) { ok = false; break; }
          if (!landed(2 * j + 1)) { ok = false; break; }
          const uint64_t b = dv + (uint64_t)(((2 * j + 1) % TP_SLOTS) * (TILE_BYTES >> 4));
          const int k_steps = (tile_len(j) + 15) / 16;               // 16-token steps that hold at least one visible key
          for (int x = 0; x < heads; ++x) {
            if (!mbar_wait(smem_u32(&bar_p[x]), j & 1, &abort_flag, TC_BUDGET_NS)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < TC_BN / 16; ++k)
              if (k < k_steps) mma_f16_ts(tmem + 256 + x * 128, tmem + x * 128 + k * 8, b + k * 128, idesc_o, (j > 0 || k > 0) ? 1u : 0u);
            if (more) scores(x, j + 1);
          }
          if (!ok) break;
          tc_commit(smem_u32(&bar_empty[(2 * j + 1) % TP_SLOTS]));
          if (more) tc_commit(smem_u32(&bar_empty[(2 * j + 2) % TP_SLOTS]));
          else tc_commit(smem_u32(&bar_o));
        }
        if (!ok) {
          if (abort_flag == 0) report_status(p.status, ST_TIMEOUT_SMEM_FULL, 11);
          abort_flag = 1;
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    if ((warp >> 2) < heads) {
      // ---------------------------------------------------------------- softmax warps: thread <-> query row of head x
      const int x = warp >> 2, q = warp & 3, r = q * 32 + lane, head = head0 + x;
      const uint32_t lane_addr = (uint32_t)(q * 32) << 16, tm_s = tmem + x * 128 + lane_addr, tm_o = tmem + 256 + x * 128 + lane_addr;
      const int pos_r = min(pos0 + q0 + r, kvlen - 1);         // rows past the chunk are computed, finite, and never stored
      const int first_key = attn_first_key(p.r.window, p.r.chunk, pos_r);
      float m = -INFINITY, l = 0.f;
      bool ok = true;
      for (int j = 0; j < n_tiles; ++j) {
        const int n0 = tile_at(j) * TC_BN;
        if (!mbar_wait(smem_u32(&bar_s[x]), j & 1, &abort_flag, TC_BUDGET_NS)) { ok = false; break; }
        tc_fence_after();
        uint32_t sv[TC_BN];
#pragma unroll
        for (int c = 0; c < TC_BN; c += 32) tmem_ld32(tm_s + c, sv + c);
        tmem_ld_wait();
        if (CAP) {
#pragma unroll
          for (int i = 0; i < TC_BN; ++i) sv[i] = __float_as_uint(attn_cap(__uint_as_float(sv[i]), p.cap_in, p.cap_log2e));
        }
        if (n0 + TC_BN - 1 > pos0 + q0 || (n0 < last_lo && n0 + TC_BN > keep)) {      // some row of the tile sees only part of these keys
          const int limit = pos_r - n0, first = first_key - n0, until = keep - n0;
#pragma unroll
          for (int i = 0; i < TC_BN; ++i)
            if (!(i <= limit && (i >= first || i < until))) sv[i] = 0xff800000u;
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < TC_BN; i += 2) mx4[(i >> 1) & 3] = fmaxf(mx4[(i >> 1) & 3], fmaxf(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])));
        const float raw = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));                   // the scale is positive
        const float mx = CAP ? raw : raw * p.scale_log2e;
        // the running maximum only moves when it is exceeded by more than 2^8 (see above)
        const float m_new = (m == -INFINITY || mx > m + 8.f) ? fmaxf(m, mx) : m;
        const float alpha = (m == -INFINITY) ? 1.f : exp2f(m - m_new);
        const float ref = m_new == -INFINITY ? 0.f : m_new;      // (a row whose window starts in a later tile)
        if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
          for (int c = 0; c < TC_D; c += 16) {
            uint32_t ov[16];
            tmem_ld16(tm_o + c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
            tmem_st16(tm_o + c, ov);
          }
        }
        l *= alpha;
        m = m_new;
        const uint64_t scale2 = f32x2(p.scale_log2e, p.scale_log2e), ref2 = f32x2(-ref, -ref);
        uint64_t sum2[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < TC_BN; c += 32) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float x0, x1;
            const uint64_t s2 = f32x2(__uint_as_float(sv[c + i]), __uint_as_float(sv[c + i + 1]));
            f32x2_split(CAP ? f32x2_add(s2, ref2) : f32x2_fma(s2, scale2, ref2), x0, x1);
            // the row sum is taken over the rounded values, the ones the tensor cores multiply
            const __nv_bfloat162 pb = __floats2bfloat162_rn(exp2f(x0), exp2f(x1));
            const uint32_t u = *reinterpret_cast<const uint32_t*>(&pb);
            sum2[(i >> 1) & 1] = f32x2_add(sum2[(i >> 1) & 1], f32x2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)));
            pk[i >> 1] = u;
          }
          tmem_st16(tm_s + c / 2, pk);          // P over the columns of S, all of which are in registers
        }
        float r0, r1;
        f32x2_split(f32x2_add(sum2[0], sum2[1]), r0, r1);
        l += r0 + r1;
        if (x == 0 && n0 + TC_BN > kv_hi) {
          // rows of V past the context in the tile's last 16-token step are zeroed, so that 0 * garbage cannot produce a NaN (see above); the
          // second head's product comes after the first one's
          const int iv = 2 * j + 1, past = kv_hi - n0, n_rows = ((past + 15) & ~15) - past;
          if (!mbar_wait(smem_u32(&bar_full[iv % TP_SLOTS]), (iv / TP_SLOTS) & 1, &abort_flag, TC_BUDGET_NS)) { ok = false; break; }
          for (int i = r; i < n_rows * 8; i += 128) {              // 16-byte chunks of those rows, per half
            const uint32_t a = ring + (iv % TP_SLOTS) * TILE_BYTES + past * 128 + i * 16;
#pragma unroll
            for (int hf = 0; hf < HALVES; ++hf)
              asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(a + hf * TC_HALF_BYTES), "r"(0) : "memory");
          }
          fence_proxy_async_smem();
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_p[x]));
      }
      if (ok && mbar_wait(smem_u32(&bar_o), 0, &abort_flag, TC_BUDGET_NS)) {
        tc_fence_after();
        const float inv = attn_norm(m, l, attn_sink_log2(p.r, head)) * p.r.out_scale;
        __nv_bfloat16* orow = p.out + (size_t)(qrow0 + q0 + r) * p.out_ld + (size_t)head * TC_D;
#pragma unroll
        for (int c = 0; c < TC_D; c += 32) {
          uint32_t ov[32];
          tmem_ld32(tm_o + c, ov);
          tmem_ld_wait();
          if (q0 + r < qlen) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint32_t pk[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(ov[i + 2 * k]) * inv, __uint_as_float(ov[i + 2 * k + 1]) * inv);
                pk[k] = *reinterpret_cast<const uint32_t*>(&b);
              }
              *reinterpret_cast<uint4*>(orow + c + i) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
          }
        }
      } else {
        if (abort_flag == 0) report_status(p.status, ST_TIMEOUT_TMEM_FULL, 12);
        abort_flag = 1;
      }
    }
  }
  if (*(volatile int*)&abort_flag) {
    // copies that are still in flight land before the shared memory is given back
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace skein

namespace skein {

template <int TC_D, bool CAP>
static int attn_prefill_pair_go(const void* q, long long q_stride, long long q_rows, const void* kv, const AttnPrefillTcParams& p, int S, int max_q_len,
                                void* stream) {
  static PerDevice allowed;
  const cudaError_t e = allow_smem(allowed, (const void*)attn_prefill_pair_kernel<TC_D, CAP>, tp_smem(TC_D));
  if (e != cudaSuccess) return (int)e;
  CUtensorMap tmQ, tmKV;
  int rc = cached_tmap_2d(&tmQ, q, (uint64_t)q_rows, (uint64_t)q_stride, 2, TC_BM);
  if (rc != 0) return rc;
  rc = cached_tmap_2d(&tmKV, kv, (uint64_t)p.num_pages * 2 * p.Hkv * p.page_size, TC_D, 2, TC_PS);
  if (rc != 0) return rc;
  dim3 grid(p.Hkv * ((p.Hq / p.Hkv + 1) / 2), S, (max_q_len + TC_BM - 1) / TC_BM);
  attn_prefill_pair_kernel<TC_D, CAP><<<grid, TP_THREADS, tp_smem(TC_D), (cudaStream_t)stream>>>(tmQ, tmKV, p);
  return (int)cudaGetLastError();
}

static int attn_prefill_maps_go(const void* q, long long q_stride, long long q_rows, const void* kv, const AttnPrefillTcParams& p, int S, int max_q_len,
                                void* stream) {
  constexpr int smem = 3 * 2 * TC_HALF_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
  static PerDevice allowed;
  const cudaError_t e = allow_smem(allowed, (const void*)attn_prefill_maps_kernel, smem);
  if (e != cudaSuccess) return (int)e;
  CUtensorMap tmQ, tmKV;
  int rc = cached_tmap_2d(&tmQ, q, (uint64_t)q_rows, (uint64_t)q_stride, 2, TC_BM / 2);
  if (rc != 0) return rc;
  rc = cached_tmap_2d(&tmKV, kv, (uint64_t)p.num_pages * 2 * p.Hkv * p.page_size, 128, 2, TC_PS);
  if (rc != 0) return rc;
  dim3 grid((max_q_len + TC_BM / 2 - 1) / (TC_BM / 2), p.Hq, S);
  attn_prefill_maps_kernel<<<grid, TC_THREADS, smem, (cudaStream_t)stream>>>(tmQ, tmKV, p);
  return (int)cudaGetLastError();
}

}  // namespace skein

// Returns 0, a cudaError_t, or a negative code for shapes this kernel does not take (the caller then uses another kernel): head
// size 128 or 64 (D: the width of a key head; 128 with two maps), pages of whole 16-token groups, 16-byte aligned rows. Rows of out are
// out_ld apart.
extern "C" int skein_attn_prefill_window(const void* q, long long q_stride, long long q_rows, const void* kv, const int* block_table,
                                         const int* q_start, const int* q_len, const int* kv_len, void* out, long long out_ld, int* status, int S,
                                         int max_q_len, int Hq, int Hkv, int D, int page_size, int max_blocks, int num_pages,
                                         const SkeinAttnRule* rule, void* stream) {
  using namespace skein;
  if (S == 0 || max_q_len == 0) return 0;
  if ((D != 128 && D != 64) || page_size % TC_PS != 0 || Hq % Hkv != 0 || q_stride % 8 != 0 || (uintptr_t)q % 16 != 0) return -1;
  if (out_ld % 8 != 0 || (uintptr_t)out % 16 != 0 || rule->scale <= 0.f) return -1;
  if (rule->maps == 2 ? D != 128 || !rule->lam || rule->gate_ld % 8 != 0 || (uintptr_t)rule->gate % 16 != 0 : rule->maps != 1 || rule->gate) return -1;
  AttnPrefillTcParams p;
  p.block_table = block_table; p.q_start = q_start; p.q_len = q_len; p.kv_len = kv_len;
  p.out = (__nv_bfloat16*)out; p.status = status; p.out_ld = out_ld; p.r = *rule;
  p.Hq = Hq; p.Hkv = Hkv; p.max_blocks = max_blocks; p.num_pages = num_pages; p.page_size = page_size;
  p.scale_log2e = rule->scale * 1.4426950408889634f;
  p.cap_log2e = rule->softcap * 1.4426950408889634f;
  p.cap_in = rule->softcap > 0.f ? 2.f * p.scale_log2e / rule->softcap : 0.f;
  auto go = [&](auto fn) { return fn(q, q_stride, q_rows, kv, p, S, max_q_len, stream); };
  if (rule->maps == 2) return rule->softcap > 0.f ? -1 : go(attn_prefill_maps_go);
  if (rule->softcap > 0.f) return D == 64 ? go(attn_prefill_pair_go<64, true>) : go(attn_prefill_pair_go<128, true>);
  return D == 64 ? go(attn_prefill_pair_go<64, false>) : go(attn_prefill_pair_go<128, false>);
}

extern "C" int skein_attn_prefill_tc(const void* q, long long q_stride, long long q_rows, const void* kv, const int* block_table,
                                     const int* q_start, const int* q_len, const int* kv_len, void* out, int* status, int S,
                                     int max_q_len, int Hq, int Hkv, int D, int page_size, int max_blocks, int num_pages,
                                     float scale, void* stream) {
  if (D != 128 || page_size != 16) return -1;
  SkeinAttnRule rule{};
  rule.maps = 1; rule.scale = scale; rule.out_scale = 1.f;
  return skein_attn_prefill_window(q, q_stride, q_rows, kv, block_table, q_start, q_len, kv_len, out, (long long)Hq * D, status, S, max_q_len, Hq,
                                   Hkv, D, page_size, max_blocks, num_pages, &rule, stream);
}
