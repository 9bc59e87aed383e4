// Causal attention of prompt portions with value heads of 128 numbers on the 5th-generation tensor cores (tcgen05).
//
// A block works on two tiles A and B of 128 query rows each that read the same keys and values: the same tokens of two heads that share
// a key head, or (`pair_heads` 0) 256 consecutive tokens of one head.  Keys and values come 64 at a time by TMA, in chunks of 64 numbers
// (128-byte swizzle).  S = Q K^T (128 x 64, float32) is made in tensor memory, in two buffers per tile of rows, so that the next scores are there
// when a softmax ends; the four softmax warps of a tile have a row to a thread, hold its 64 scores in registers (no exchange between
// threads) and write the weights, rounded to the operands' 16-bit type, over S's columns, from where
// they enter O += P V as the first operand: they never pass through shared memory.  O (128 x 128, float32) stays in tensor memory; a warp
// scales its rows' O where one of their maxima has grown.
//
// Keys have KC chunks of 64 numbers.  Two sources: a paged cache (pages found through the block table; positions on no page are read
// behind the pages' end as zeros), or rows side by side (latent_expand.cu), request after request, whose third chunk, a part that all
// heads share, comes from pages.  From both, the values of positions behind the block's last row are wiped: they may be anything, another
// request's not-a-numbers too.  F16: queries, keys, weights and values are float16
// (the shared third chunk bfloat16 on both sides), with a factor per row and head on the scores (q_scale), one per head on the values
// (v_scale), and weights 2^14 times as large, which leaves 28 powers of two of full precision below the largest; else bfloat16.
//
// Warps 0-3: rows of tile A, 4-7: of tile B; 8: TMA; 9 and 10: MMA issue of A and of B (9: tensor memory).  One block to a multiprocessor (192 or 224 KB).  Every wait
// is bounded; one that runs out records its code, and the block ends when its copies have landed.
//
// What bounds it: per 64 keys a pair of tiles takes 1,024 clocks of the special-function unit (16 exponentials a clock), about 1,300 issue slots a
// scheduler (the scaling of O is a third of them) and 2 x 640 clocks of tensor core (2 x 832 with three chunks); it takes 2,650 clocks, the
// softmax threads' chain of one step after the other.  3,900 clocks pass from the grid's start to the first product's
// end (queries and keys of all blocks at once) and 3,700 behind the last one.  The instructions are fetched by far more code than the
// first-level caches hold, so every loop is as short as it can be: unrolled copies of the waits and products alone had made it 25 us.
// Measured, 16 heads over 4 key heads of 128: 2 prompts of 1,024 tokens in chunks of 512 53 -> 19.4 us (mma.sync form, this), the layer of width 2,048
// 120.5 -> 85.8; 1 prompt of 1,024 63 -> 28; 128 rows 12.0 -> 9.8.
#include <cuda.h>
#include <cuda_fp16.h>
#include <math.h>

#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int ROWS = 128, KEYS = 64, VD = 128;
constexpr uint32_t CHUNK = ROWS * 128, K_CHUNK = KEYS * 128;      // 128 rows, 64 keys x 64 numbers of 16 bits
constexpr int SOFT_WARPS = 8, THREADS = (SOFT_WARPS + 3) * 32;
constexpr int stages(int kc) { return kc == 2 ? 4 : 3; }         // of keys and of values
constexpr size_t smem_bytes(int kc) { return (size_t)2 * kc * CHUNK + (size_t)stages(kc) * (kc + 2) * K_CHUNK + 512; }

struct WideArgs {
  __nv_bfloat16* out;            // [T, H * 128]
  const int* table;              // [R, table_stride]
  const int* req_q_start;        // [R + 1]
  const int* req_pos0;           // [R]
  const float* sinks;            // [H] or null: the score of one more key without a value
  const float* gate;             // float32 rows or null: the output is multiplied by sigmoid of the row's number at h * gate_head + d * gate_col
  const float* q_scale;          // [T, H] or null: the factor of a row's scores
  const float* v_scale;          // F16: [H], the factor that a head's values carry
  int* error;
  long long gate_stride;
  int gate_head, gate_col;
  int side_by_side;              // keys and values lie side by side, request after request (latent_expand.cu), instead of in pages
  int table_stride, num_req, H, heads_per_key, v_head0, page_shift, rows_end, window, chunk, pair_heads;
  float scale_log2;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <bool F16>
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  if (!F16) return pack_bf16(lo, hi);
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int KC, bool F16>
__global__ void __launch_bounds__(THREADS, 1)
attention_wide_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q2, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_shared, WideArgs args) {
  constexpr int ST = stages(KC);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t q_tile = base, k_tile = q_tile + 2 * KC * CHUNK, v_tile = k_tile + ST * KC * K_CHUNK, bars = v_tile + ST * 2 * K_CHUNK;
  const uint32_t q_full = bars, k_full = bars + 16, k_empty = k_full + 8 * ST, v_full = k_empty + 8 * ST, v_empty = v_full + 8 * ST,
                 s_full = v_empty + 8 * ST, p_full = s_full + 32, pv_done = p_full + 32, wiped = pv_done + 16, tmem_slot = wiped + 8;
  const int warp = warp_number(), lane = threadIdx.x & 31;

  // Which request and which of its tiles?  As in attention_tc: the last tile of every request first, then the one before it, ...: late
  // tiles see the most keys.  Every warp finds its tile for itself, 32 requests at a time.
  const int span = args.pair_heads ? ROWS : 2 * ROWS;
  int tile = blockIdx.y, req = -1, q0 = 0, q_len = 0;
  for (int r0 = 0; r0 < args.num_req && req < 0; r0 += 32) {
    const int r = r0 + lane;
    const int len = r < args.num_req ? args.req_q_start[r + 1] - args.req_q_start[r] : 0;
    const int tiles = (len + span - 1) / span;
    const int group_tiles = __reduce_add_sync(0xffffffffu, tiles);
    if (tile >= group_tiles) { tile -= group_tiles; continue; }
    for (int level = 0; req < 0; ++level) {            // ends: tile < group_tiles
      const unsigned have = __ballot_sync(0xffffffffu, tiles > level);
      const int n = __popc(have);
      if (tile < n) {
        const int src = __fns(have, 0, tile + 1);      // the lane of the (tile + 1)-th such request
        req = r0 + src;
        q_len = __shfl_sync(0xffffffffu, len, src);
        q0 = (__shfl_sync(0xffffffffu, tiles, src) - 1 - level) * span;
      } else {
        tile -= n;
      }
    }
  }
  if (req < 0) return;
  if (base & 1023u) {                                  // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicExch(args.error, 80);
    return;
  }
  // tile 0 is A, tile 1 is B: rows, first row's position, and which of the 64-key tiles from k_begin on it reads
  const int h0 = args.pair_heads ? 2 * blockIdx.x : blockIdx.x;
  const int row_first = args.req_q_start[req] + q0, pos_first = args.req_pos0[req] + q0;
  const int rows_a = min(ROWS, q_len - q0), rows_b = args.pair_heads ? rows_a : max(0, min(ROWS, q_len - q0 - ROWS));
  const int pos_a = pos_first, pos_b = args.pair_heads ? pos_first : pos_first + ROWS;
  auto first_key = [&](int pos) {
    const int from_window = args.window > 0 ? max(0, pos - args.window + 1) : 0;
    return args.chunk > 0 ? max(from_window, pos / args.chunk * args.chunk) : from_window;
  };
  const int k_begin = first_key(pos_a) / KEYS * KEYS;
  const int last_key = max(pos_a + rows_a, rows_b > 0 ? pos_b + rows_b : 0) - 1;
  const int end_a = (pos_a + rows_a - 1 - k_begin) / KEYS + 1;
  const int start_b = rows_b > 0 ? (first_key(pos_b) - k_begin) / KEYS : 0;
  const int end_b = rows_b > 0 ? (pos_b + rows_b - 1 - k_begin) / KEYS + 1 : 0;
  const bool wipes = (last_key - k_begin + 1) % KEYS != 0;      // the last tile holds positions behind the last row's (side by side: the next request's too)
  const int num_tiles = max(end_a, end_b);             // no tile is read by neither: B's first key is at most the one behind A's last

  if (threadIdx.x == 0) {
    mbar_init(wiped, 1);
    for (int i = 0; i < ST; ++i) {
      mbar_init(k_full + 8 * i, 1); mbar_init(k_empty + 8 * i, 2);        // both tiles' issuing threads are through with it
      mbar_init(v_full + 8 * i, 1); mbar_init(v_empty + 8 * i, 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full + 8 * i, 1);
      mbar_init(pv_done + 8 * i, 1);
    }
    for (int i = 0; i < 4; ++i) {                      // a tile's two buffers of S: the one may be filled, or weighed, before the other's has been looked at
      mbar_init(s_full + 8 * i, 1); mbar_init(p_full + 8 * i, SOFT_WARPS / 2);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == SOFT_WARPS && lane < 5) {
    const CUtensorMap* map = lane == 0 ? &map_q : lane == 1 ? &map_k : lane == 2 ? &map_v : lane == 3 ? &map_q2 : &map_shared;
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
  }
  if (warp == SOFT_WARPS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*(volatile uint32_t*)(smem_raw + (tmem_slot - base)));      // columns: two S of A, two S of B, O of A, O of B

  if (warp == SOFT_WARPS) {
    // ---- TMA
    const int* my_table = args.table + (size_t)req * args.table_stride;
    const int box = min(KEYS, 1 << args.page_shift), boxes = KEYS / box;
    const bool paged = !args.side_by_side;
    int k_row0 = 0;                                    // the row of key 0 (rows start at a request's first visible 64 keys)
    if (!paged) {
      auto from = [&](int r) { return args.window > 0 ? max(0, args.req_pos0[r] - args.window + 1) / KEYS * KEYS : 0; };
      for (int r = lane; r < req; r += 32) k_row0 += args.req_pos0[r] - from(r) + args.req_q_start[r + 1] - args.req_q_start[r];
      k_row0 = (int)__reduce_add_sync(0xffffffffu, (unsigned)k_row0) - from(req);
    }
    const int kh = args.pair_heads || args.heads_per_key > 1 ? h0 / args.heads_per_key : h0;
    auto cell_of = [&](int t) {                        // lane i: where the i-th box of tile t lies in the pages
      const int k = k_begin + t * KEYS + lane * box;
      const int page = lane < boxes && k <= last_key ? my_table[k >> args.page_shift] : 0;
      return page > 0 ? (page << args.page_shift) + (k & ((1 << args.page_shift) - 1)) : args.rows_end;
    };
    auto arm = [&](uint32_t full, uint32_t empty, int use, uint32_t bytes) -> bool {      // the use-th copy into this place
      bool fine = true;
      if (lane == 0) {
        if (use > 0) fine = mbar_wait_short(empty, (uint32_t)(use - 1) & 1u, args.error, 81);
        if (fine) mbar_expect_tx(full, bytes);
      }
      return __shfl_sync(0xffffffffu, fine ? 1 : 0, 0) != 0;
    };
    auto bring_k = [&](int t, int cell) -> bool {
      const uint32_t full = k_full + 8 * (t % ST), to = k_tile + (uint32_t)(t % ST) * KC * K_CHUNK;
      if (!arm(full, k_empty + 8 * (t % ST), t / ST, KC * K_CHUNK)) return false;
      if (paged) {
        if (lane < boxes)
          for (int c = 0; c < KC; ++c) tma_load_3d(to + c * K_CHUNK + (uint32_t)(lane * box) * 128u, &map_k, c * 64, kh, cell, full);
      } else {
        if (lane < 2) tma_load_3d(to + lane * K_CHUNK, &map_k, lane * 64, kh, k_row0 + k_begin + t * KEYS, full);
        if (KC == 3 && lane < boxes) tma_load_3d(to + 2 * K_CHUNK + (uint32_t)(lane * box) * 128u, &map_shared, 0, 0, cell, full);
      }
      return true;
    };
    auto bring_v = [&](int t, int cell) -> bool {
      const uint32_t full = v_full + 8 * (t % ST), to = v_tile + (uint32_t)(t % ST) * 2 * K_CHUNK;
      if (!arm(full, v_empty + 8 * (t % ST), t / ST, 2 * K_CHUNK)) return false;
      if (paged) {
        if (lane < boxes)
          for (int c = 0; c < 2; ++c) tma_load_3d(to + c * K_CHUNK + (uint32_t)(lane * box) * 128u, &map_v, c * 64, kh, cell, full);
      } else if (lane < 2) {
        tma_load_3d(to + lane * K_CHUNK, &map_v, lane * 64, args.v_head0 + kh, k_row0 + k_begin + t * KEYS, full);
      }
      return true;
    };
    const int q_tiles = rows_b > 0 ? 2 : 1;
    int cell = cell_of(0);                             // the table is the step's own data, uploaded before it
    pdl_wait();
    auto bring_q = [&](int x) {
      if (lane == 0) mbar_expect_tx(q_full + 8 * x, KC * CHUNK);
      __syncwarp();
      if (lane < KC) {
        const int h = h0 + (args.pair_heads ? x : 0), row = row_first + (args.pair_heads ? 0 : x * ROWS);
        const uint32_t to = q_tile + (uint32_t)(x * KC + lane) * CHUNK;
        if (F16 && lane == 2) tma_load_2d(to, &map_q2, h * 64, row, q_full + 8 * x);
        else tma_load_2d(to, &map_q, (h * (F16 ? 2 : KC) + lane) * 64, row, q_full + 8 * x);
      }
    };
    // in the order of their use: the queries of A, the first keys, the queries of B, then keys two tiles ahead of values
    bring_q(0);
    bool ok = bring_k(0, cell);
    int k_issued = ok ? 1 : 0, v_issued = 0;
    if (q_tiles == 2) bring_q(1);
    int later = 0;                                     // the boxes of tile k_issued - 1
    auto bring_next_k = [&]() {
      later = cell_of(k_issued);
      ok = bring_k(k_issued, later);
      if (ok) ++k_issued;
    };
    if (ok && num_tiles > 1) bring_next_k();
    for (int t = 0; t < num_tiles && ok; ++t) {
      const int now = cell;
      cell = later;
      if (t + 2 < num_tiles) bring_next_k();
      if (ok) ok = bring_v(t, now);
      if (ok) v_issued = t + 1;
    }
    if (ok && wipes) {
      // positions behind the last row's are nobody's yet, or (side by side) another request's: what their places hold enters P V times
      // zero, so it has to be finite
      const int t = num_tiles - 1, live = last_key - (k_begin + t * KEYS) + 1;
      if (lane == 0) ok = mbar_wait_short(v_full + 8 * (t % ST), (uint32_t)(t / ST) & 1u, args.error, 85);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      uint8_t* at = smem_raw + (v_tile - base) + (uint32_t)(t % ST) * 2 * K_CHUNK;
      for (int i = lane; ok && i < 2 * (KEYS - live) * 8; i += 32) {
        const int c = i / ((KEYS - live) * 8), rest = i - c * ((KEYS - live) * 8);
        *reinterpret_cast<uint4*>(at + c * K_CHUNK + (live + (rest >> 3)) * 128 + (rest & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(wiped);
    }
    if (!ok && lane == 0) {                            // nobody may be consuming any more: wait for the copies in flight
      for (int x = 0; x < q_tiles; ++x) mbar_wait_short(q_full + 8 * x, 0u, args.error, 82);
      for (int t = max(0, k_issued - ST); t < k_issued; ++t) mbar_wait_short(k_full + 8 * (t % ST), (uint32_t)(t / ST) & 1u, args.error, 82);
      for (int t = max(0, v_issued - ST); t < v_issued; ++t) mbar_wait_short(v_full + 8 * (t % ST), (uint32_t)(t / ST) & 1u, args.error, 82);
    }
    __syncwarp();
  } else if (warp > SOFT_WARPS) {
    // ---- MMA issue, a thread to each tile of rows: P V per tile of keys, then S two tiles on, into the columns that those weights have left.
    // Short code and loops that are not unrolled: the thread's instructions come between those of two softmax warps and are fetched
    // anew each time.  (With every product laid out by itself and a whole warp to vote on every wait 64 keys took 4,300 clocks; with
    // one thread for both tiles, 2,700.)
    constexpr uint32_t IDESC_16 = F16 ? make_idesc_f16(ROWS, KEYS) : make_idesc(ROWS, KEYS), IDESC_SHARED = make_idesc(ROWS, KEYS);
    constexpr uint32_t IDESC_O = F16 ? make_idesc_f16(ROWS, VD, 1) : make_idesc(ROWS, VD, 1);
    const uint32_t x = (uint32_t)(warp - SOFT_WARPS - 1);
    const int n = (int)uniform((uint32_t)num_tiles), start = (int)uniform((uint32_t)(x ? start_b : 0)), end = (int)uniform((uint32_t)(x ? end_b : end_a));
    const bool wiping = uniform(wipes ? 1u : 0u) != 0;
    pdl_wait();
    if (elect_one()) {
      bool ok = true;
      auto wait = [&](uint32_t bar, int use, int code) {
        if (ok) ok = mbar_wait_short(bar, (uint32_t)use & 1u, args.error, code);
      };
      const uint64_t da = make_desc(q_tile + x * KC * CHUNK);
      int k_st = 0, k_use = 0, v_st = 0, v_use = 0;    // the next tile's places, and how often they have been used
#pragma unroll 1
      for (int t = -2; t < n && ok; ++t) {
        if (t >= 0) {
          wait(v_full + 8 * v_st, v_use, 85);
          if (t >= start && t < end) {
            const int local = t - start, half = local & 1;
            if (wiping && t + 1 == n) wait(wiped, 0, 87);
            wait(p_full + 8 * (2 * x + half), local >> 1, 86);
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = make_desc_mn(v_tile + (uint32_t)v_st * 2 * K_CHUNK, K_CHUNK);
            const uint32_t d = tmem + 256u + 128u * x, pa = tmem + 128u * x + 64u * half;
#pragma unroll
            for (int k = 0; k < KEYS / 16; ++k) umma_ts(d, pa + 8u * k, db + (uint64_t)(k * (2048 >> 4)), IDESC_O, k > 0 ? 1u : (uint32_t)local);
            umma_commit(pv_done + 8 * x);
            umma_commit(v_empty + 8 * v_st);
          } else if (ok) {
            mbar_arrive(v_empty + 8 * v_st);
          }
          if (++v_st == ST) { v_st = 0; ++v_use; }
        }
        if (t + 2 < n) {
          wait(k_full + 8 * k_st, k_use, 84);
          if (t + 2 >= start && t + 2 < end) {
            const int local = t + 2 - start, half = local & 1;
            if (local == 0) wait(q_full + 8 * x, 0, 83);
            if (local >= 2) wait(pv_done + 8 * x, local, 88);          // the weights of two tiles before lie in these columns
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = make_desc(k_tile + (uint32_t)(k_st * KC) * K_CHUNK);
            const uint32_t d = tmem + 128u * x + 64u * half;
#pragma unroll
            for (int c = 0; c < KC; ++c)
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma(d, da + (uint64_t)(c * (CHUNK >> 4) + 2 * k), db + (uint64_t)(c * (K_CHUNK >> 4) + 2 * k), F16 && c == 2 ? IDESC_SHARED : IDESC_16,
                     c > 0 || k > 0 ? 1u : 0u);
            umma_commit(s_full + 8 * (2 * x + half));
            umma_commit(k_empty + 8 * k_st);
          } else if (ok) {
            mbar_arrive(k_empty + 8 * k_st);
          }
          if (++k_st == ST) { k_st = 0; ++k_use; }
        }
      }
    }
    __syncwarp();
  } else {
    // ---- softmax: TMEM lane = row
    const int x = warp >> 2, r = (warp & 3) * 32 + lane;
    const int rows = x == 0 ? rows_a : rows_b, start = x == 0 ? 0 : start_b, end = x == 0 ? end_a : end_b;
    const int h = h0 + (args.pair_heads ? x : 0);
    const int row = row_first + (args.pair_heads ? 0 : x * ROWS) + r;
    const bool live = r < rows;
    const int qpos = (x == 0 ? pos_a : pos_b) + r;
    const int qlow = first_key(qpos);
    const uint32_t s_first = tmem + 128u * x + ((uint32_t)((warp & 3) * 32) << 16), o_at = s_first + 256u;
    const float v_scale = F16 ? args.v_scale[h] : 1.f;
    pdl_wait();
    const float scale = args.scale_log2 * (args.q_scale && live ? args.q_scale[(size_t)row * args.H + h] : 1.f);
    constexpr float UP = F16 ? 14.f : 0.f;             // the weights and their sum are 2^UP times what they are
    float m_run = -INFINITY, l = 0.f;
    if (args.sinks) {
      m_run = args.sinks[h] * 1.4426950408889634f;
      l = F16 ? 16384.f : 1.f;
    }
    bool ok = true;
    for (int t = start; t < end; ++t) {
      const int local = t - start, k0 = k_begin + t * KEYS, buffer = 2 * x + (local & 1);
      const uint32_t s_at = s_first + 64u * (local & 1);
      if (lane == 0) ok = mbar_wait_short(s_full + 8 * buffer, (uint32_t)(local >> 1) & 1u, args.error, 89);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      tc_fence_after();
      uint32_t s[KEYS];
#pragma unroll
      for (int c = 0; c < KEYS; c += 32) tmem_ld32(s_at + c, s + c);
      tmem_ld_wait();
      // this row sees the keys lo <= j < hi of the tile
      const int hi = live ? min(KEYS, qpos - k0 + 1) : 0, lo = max(0, qlow - k0);
      float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (!__all_sync(0xffffffffu, lo == 0 && hi == KEYS)) {
#pragma unroll
        for (int j = 0; j < KEYS; ++j) s[j] = j >= lo && j < hi ? s[j] : 0xff800000u;      // minus infinity
      }
#pragma unroll
      for (int j = 0; j < KEYS; ++j) top[j & 3] = fmaxf(top[j & 3], __uint_as_float(s[j]));
      const float m_tile = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * scale;      // the scale is positive: the maximum commutes with it
      const float m_new = fmaxf(m_run, m_tile);
      const bool grown = __any_sync(0xffffffffu, m_new > m_run);
      const float alpha = m_new > -INFINITY ? fast_exp2(m_run - m_new) : 1.f;        // 2^(-inf) = 0 before the first visible key
      m_run = m_new;
      const float m = m_run > -INFINITY ? m_run - UP : 0.f;  // nothing seen yet: every weight is 2^(-inf) = 0
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < KEYS; j += 2) {
        const float p0 = fast_exp2(fmaf(__uint_as_float(s[j]), scale, -m)), p1 = fast_exp2(fmaf(__uint_as_float(s[j + 1]), scale, -m));
        sum[(j >> 1) & 3] += p0 + p1;
        s[j >> 1] = pack<F16>(p0, p1);
      }
      l = fmaf(l, alpha, (sum[0] + sum[1]) + (sum[2] + sum[3]));
      tmem_st32(s_at, s);
      // O's scale moves when the product of the tile before is through, which has had the time of the exponentials.  (Every phase of
      // the barrier is waited for, also where no maximum has grown: a wait two phases ahead would be answered at once.  Four more warps
      // that scale O for the softmax warps were no faster: P V, the scaling and the next P V follow one another either way.)
      if (local > 0) {
        if (lane == 0) ok = mbar_wait_short(pv_done + 8 * x, (uint32_t)(local - 1) & 1u, args.error, 91);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
        if (grown) {
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < VD; c += 32) {
            uint32_t o[32];
            tmem_ld32(o_at + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tmem_st32(o_at + c, o);
          }
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + 8 * buffer);
    }
    if (ok && end > start) {
      if (lane == 0) ok = mbar_wait_short(pv_done + 8 * x, (uint32_t)(end - start - 1) & 1u, args.error, 90);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (ok) {
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / (l * v_scale) : 0.f;
        // through this tile's place of the queries (its products are done), so that a warp stores whole rows of 256 bytes: a
        // piece of 16 bytes lies at its number XOR the low bits of its row
        uint8_t* stage = smem_raw + (uint32_t)x * KC * CHUNK + (uint32_t)(warp & 3) * 32 * 256;
        const float* gate = args.gate && live ? args.gate + (size_t)row * args.gate_stride + (size_t)h * args.gate_head : nullptr;
#pragma unroll 1
        for (int c = 0; c < VD; c += 32) {
          uint32_t o[32];
          tmem_ld32(o_at + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(o[j + e]) * inv;
            if (gate)
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = __fdividef(v[e], 1.f + __expf(-gate[(c + j + e) * args.gate_col]));
            *reinterpret_cast<uint4*>(stage + lane * 256 + ((((c + j) >> 3) ^ (lane & 7)) << 4)) =
                make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
          }
        }
        __syncwarp();
        const int first = row - lane, most = rows - (warp & 3) * 32;
#pragma unroll 4
        for (int i = lane >> 4; i < 32 && i < most; i += 2) {
          const uint4 v = *reinterpret_cast<const uint4*>(stage + i * 256 + (((lane & 15) ^ (i & 7)) << 4));
          *reinterpret_cast<uint4*>(args.out + ((size_t)(first + i) * args.H + h) * VD + (lane & 15) * 8) = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == SOFT_WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ------------------------------------------------------------------- host --

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
int* g_error_host = nullptr;
int* g_error_dev = nullptr;
std::mutex g_mutex;
AykPerDevice g_configured;

int setup() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (err != cudaSuccess || fn == nullptr || q != cudaDriverEntryPointSuccess)
      return ayk_fail("ayk_attention_wide_tc: cuTensorMapEncodeTiled is not available from this driver");
    g_encode = (EncodeTiledFn)fn;
  }
  if (!g_error_host) {
    cudaError_t err = cudaHostAlloc((void**)&g_error_host, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (err != cudaSuccess) return ayk_fail("ayk_attention_wide_tc: cudaHostAlloc: %s", cudaGetErrorString(err));
    *g_error_host = 0;
    err = cudaHostGetDevicePointer((void**)&g_error_dev, g_error_host, 0);
    if (err != cudaSuccess) return ayk_fail("ayk_attention_wide_tc: cudaHostGetDevicePointer: %s", cudaGetErrorString(err));
  }
  if (!g_configured.here()) {
    cudaError_t err = cudaFuncSetAttribute(attention_wide_tc_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(2));
    if (err == cudaSuccess) err = cudaFuncSetAttribute(attention_wide_tc_kernel<3, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(3));
    if (err != cudaSuccess) return ayk_fail("ayk_attention_wide_tc: shared memory %zu: %s", smem_bytes(3), cudaGetErrorString(err));
    g_configured.here() = true;
  }
  return 0;
}

// [rows][heads][width] 16-bit numbers; a box is box_rows rows x 64 numbers of one head, 128-byte swizzle.
int encode(CUtensorMap* map, const void* ptr, long long rows, int heads, int width, int box_rows, bool f16) {
  cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)heads, (cuuint64_t)rows};
  cuuint64_t strides[2] = {(cuuint64_t)width * 2, (cuuint64_t)heads * width * 2};
  cuuint32_t box[3] = {64u, 1u, (cuuint32_t)box_rows};
  cuuint32_t elem[3] = {1, 1, 1};
  CUresult r = g_encode(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return ayk_fail("ayk_attention_wide_tc: cuTensorMapEncodeTiled failed with %d (rows %lld, %d heads of %d)", (int)r, rows, heads, width);
  return 0;
}
// [rows][width] 16-bit numbers; a box is 128 rows x 64 numbers.
int encode_rows(CUtensorMap* map, const void* ptr, long long rows, int width, bool f16) {
  cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)width * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)ROWS};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = g_encode(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return ayk_fail("ayk_attention_wide_tc: cuTensorMapEncodeTiled failed with %d (rows %lld of %d)", (int)r, rows, width);
  return 0;
}

int page_shift_of(int page_size) {
  int shift = 0;
  while ((1 << shift) < page_size) ++shift;
  return (1 << shift) == page_size ? shift : -1;
}

}  // namespace

AYK_EXPORT int ayk_attention_wide_tc_error() { return g_error_host ? *g_error_host : 0; }

// Whether the kernel takes grouped heads of this size over this cache: heads of 128, pages of a power of two from the swizzle's 8 rows on.
AYK_EXPORT int ayk_attention_wide_tc_takes(int DK, int DV, int pages, int page_size, const void* q, const void* kcache, const void* vcache) {
  if (DK != 128 || DV != 128 || page_size < 8 || page_shift_of(page_size) < 0 || (long long)pages * page_size >= (1ll << 31)) return 0;
  return ((uintptr_t)q | (uintptr_t)kcache | (uintptr_t)vcache) % 16 == 0;
}

// out [T, H * 128], q [T, H * 128] bfloat16; caches [pages, page_size, G, 128] bfloat16; head h reads key and value head h / (H / G).  A query
// sees the keys at its own position and before it, with a window or a chunk as the grouped attention has them.  sinks [H] or null; gate float32
// rows of gate_stride, H * 128 used, or null.
AYK_EXPORT int ayk_attention_wide_tc(void* out, const void* q, const void* kcache, const void* vcache, int pages, const int* table, int table_stride,
                                     const int* req_q_start, const int* req_pos0, int num_req, int total_rows, int H, int G, int page_size, float scale,
                                     const float* sinks, int window, int chunk, const float* gate, long long gate_stride, cudaStream_t stream) {
  if (num_req == 0 || total_rows == 0) return 0;
  AYK_REQUIRE(ayk_attention_wide_tc_takes(128, 128, pages, page_size, q, kcache, vcache) && (uintptr_t)out % 16 == 0,
              "ayk_attention_wide_tc: pages of %d, or the operands' alignment, are not taken", page_size);
  AYK_REQUIRE(G >= 1 && H % G == 0, "ayk_attention_wide_tc: %d heads cannot share %d key heads", H, G);
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (setup() != 0) return -1;
  }
  const int shift = page_shift_of(page_size), box = page_size < KEYS ? page_size : KEYS;
  const long long cells = (long long)pages * page_size;
  CUtensorMap mq, mk, mv;
  if (encode_rows(&mq, q, total_rows, H * 128, false) || encode(&mk, kcache, cells, G, 128, box, false) || encode(&mv, vcache, cells, G, 128, box, false)) return -1;
  const int pair = (H / G) % 2 == 0 ? 1 : 0, span = pair ? ROWS : 2 * ROWS;
  WideArgs args{(__nv_bfloat16*)out, table, req_q_start, req_pos0, sinks, gate, nullptr, nullptr, g_error_dev, gate_stride, 128, 1, 0,
                table_stride, num_req, H, H / G, 0, shift, (int)cells, window, chunk, pair, scale * 1.4426950408889634f};
  AYK_REQUIRE(total_rows / span + num_req <= 65535, "ayk_attention_wide_tc: too many row tiles (%d rows, %d requests)", total_rows, num_req);
  ayk_launch(attention_wide_tc_kernel<2, false>, dim3(pair ? H / 2 : H, total_rows / span + num_req), dim3(THREADS), smem_bytes(2), stream, mq, mq, mk, mv, mk, args);
  return ayk_check_launch("ayk_attention_wide_tc");
}

// The expanded latent attention: out [T, H * 128] bfloat16; q16, q_rot, q_scale as latent_expand.cu makes them; kv [kv_rows, 2 H, 128] float16, keys of
// every head and then values, which carry the factor v_scale [H]; rope_pages [pages, page_size, 64] bfloat16, shared by the heads.  gate: float32 rows of gate_stride, the number at
// h * gate_head + d * gate_col, or null.
AYK_EXPORT int ayk_attention_expanded_tc(void* out, const void* q16, const void* q_rot, const float* q_scale, const float* v_scale, const void* kv, int kv_rows, const void* rope_pages,
                                         int pages, const int* table, int table_stride, const int* req_q_start, const int* req_pos0, int num_req,
                                         int total_rows, int H, int page_size, float scale, int window, const float* gate, long long gate_stride,
                                         int gate_head, int gate_col, cudaStream_t stream) {
  if (num_req == 0 || total_rows == 0) return 0;
  AYK_REQUIRE(page_size >= 8 && page_shift_of(page_size) >= 0 && (long long)pages * page_size < (1ll << 31) && scale > 0.f && H >= 1,
              "ayk_attention_expanded_tc: pages of %d are not taken", page_size);
  AYK_REQUIRE((((uintptr_t)out | (uintptr_t)q16 | (uintptr_t)q_rot | (uintptr_t)kv | (uintptr_t)rope_pages) & 15) == 0, "ayk_attention_expanded_tc: operands must be 16-byte aligned");
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (setup() != 0) return -1;
  }
  const int shift = page_shift_of(page_size), box = page_size < KEYS ? page_size : KEYS;
  const long long cells = (long long)pages * page_size;
  CUtensorMap mq, mr, mkv, ms;
  if (encode_rows(&mq, q16, total_rows, H * 128, true) || encode_rows(&mr, q_rot, total_rows, H * 64, false) ||
      encode(&mkv, kv, kv_rows, 2 * H, 128, KEYS, true) || encode(&ms, rope_pages, cells, 1, 64, box, false)) return -1;
  WideArgs args{(__nv_bfloat16*)out, table, req_q_start, req_pos0, nullptr, gate, q_scale, v_scale, g_error_dev, gate_stride, gate_head, gate_col, 1,
                table_stride, num_req, H, 1, H, shift, (int)cells, window, 0, 0, scale * 1.4426950408889634f};
  AYK_REQUIRE(total_rows / (2 * ROWS) + num_req <= 65535, "ayk_attention_expanded_tc: too many row tiles (%d rows, %d requests)", total_rows, num_req);
  ayk_launch(attention_wide_tc_kernel<3, true>, dim3(H, total_rows / (2 * ROWS) + num_req), dim3(THREADS), smem_bytes(3), stream, mq, mr, mkv, mkv, ms, args);
  return ayk_check_launch("ayk_attention_expanded_tc");
}
