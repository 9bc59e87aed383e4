// Latent attention of prompt portions on the 5th-generation tensor cores (tcgen05), bfloat16 pages.
//
// The arithmetic of latent_mma.cu: a head's query is [U_k^T q_n ; q_r] (rank + rot numbers), a key is the cached pair
// [c ; k_r], the weighted sum runs over c, all heads share the keys.  A CTA takes 128 (row, head) pairs of one request (BR
// consecutive rows times HG heads) and, for latents wider than 256, one half of O's columns:
//   S = Q K^T   M = 128 pairs, N = 32 keys, K = rank + rot; Q stays in shared memory (bfloat16, up to 144 KB)
//   online softmax in 32-bit, a thread per pair; P as bfloat16 into shared memory
//   O += P C    M = 128, N = the CTA's columns of the latent (up to 256), accumulated in tensor memory
// O of all 512 columns would fill tensor memory and leave no room for S, so two CTAs make the same scores, each for its
// half of the columns: (576 + 256) / (576 + 512) of the products twice, against an exchange between CTAs per tile.
//
// A key tile is 32 positions in chunks of 64 numbers (4 KB, 128-byte swizzle), two tiles in shared memory.  The chunks whose
// columns the CTA does not sum ("foreign": the other half and the rotated part) are free once S is made, its own ones only
// behind P C, so the MMA warp issues: foreign part of S(t + 1), P C of tile t, own part of S(t + 1).  The softmax of tile t
// runs under the foreign part, and a buffer that P C gives back has a whole tile's products to be filled again.
//
// A warp whose rows' maxima have all stayed where they were leaves O, in tensor memory, as it is; else it scales its rows.
// (Moving the weights' reference only when a maximum has grown by 2^8 made the error against 64 bits 1.5 to 4 % larger, more
// for short contexts: the largest weight is 1, which bfloat16 holds exactly, only while the reference is the maximum.)
//
// Warps 0..3: softmax, a TMEM lane (pair) per thread, and the output; warp 4: TMA producer (a box per lane); warp 5: MMA
// issue and TMEM allocation.  All warps convert the queries first.  Every mbarrier wait is bounded; one that runs out
// records a code and the CTA winds down.
// Measured, 1,024 + 777 rows of 16 heads, latent 512 + 64, no window: the layer 452 -> 356 us (mma.sync before: 286 us of it), and with
// the chunk counts as constants (straight lines of MMAs) 288 -> 272, this kernel then 167; with the reference at the
// maximum always 281.
#include <cuda.h>
#include <math.h>

#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int AQ = 128;               // pairs per CTA
constexpr int NK = 32;                // keys per tile
constexpr int MAX_CHUNKS = 9;         // runs of 64 numbers of a key: 512 + 64
constexpr int Q_CHUNK = AQ * 128, K_CHUNK = NK * 128, P_BYTES = AQ * NK * 2;
constexpr int THREADS = 192;
// Tensor memory: O in columns 0 .. 64 own - 1, two buffers of 32 for S behind it; the next power of two is asked for.
__host__ __device__ constexpr uint32_t tmem_columns(int own) { return own <= 1 ? 128u : (own <= 3 ? 256u : 512u); }

struct LatentArgs {
  float* out;                         // [T, H, rank]
  const float* query;                 // [T, H, rank + rot]
  const int* table;
  const int* req_q_start;
  const int* req_pos0;
  int* error;
  int table_stride, num_req, H, HG, BR, rank, rot, page_shift, window, own;      // own: chunks whose columns a CTA sums
  int rows_end;                       // rows of the pages: a copy from there on brings zeros
  int two_halves;                     // 1: a CTA sums one half of the latent's columns; blocks 2 i and 2 i + 1 are tile i's
  float scale_log2;
};

// Descriptor of an operand whose rows are 64 bytes (32 bfloat16 of K), 64-byte swizzle, groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t make_desc_64(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;             // SWIZZLE_64B
  return d;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// FOREIGN, OWN: chunks of either kind, constants for the usual sizes (the products are then straight lines of MMAs); 0, 0: by
// the arguments.
template <int FOREIGN, int OWN>
__global__ void __launch_bounds__(THREADS, 1)
latent_tc_kernel(const __grid_constant__ CUtensorMap map_latent, const __grid_constant__ CUtensorMap map_rope, const LatentArgs args) {
  // Tiles of the requests' last rows see the most keys: they start first (blocks are handed out in order).
  int tile = (int)(gridDim.x >> args.two_halves) - 1 - (int)(blockIdx.x >> args.two_halves), req = -1, q0 = 0, q_len = 0;
  for (int r = 0; r < args.num_req; ++r) {
    const int len = args.req_q_start[r + 1] - args.req_q_start[r];
    const int n = (len + args.BR - 1) / args.BR;
    if (tile < n) { req = r; q0 = tile * args.BR; q_len = len; break; }
    tile -= n;
  }
  if (req < 0) return;
  const int H = args.H, HG = args.HG, rank = args.rank, rot = args.rot, Dk = rank + rot;
  const int half = args.two_halves ? (int)(blockIdx.x & 1) : 0, h0 = blockIdx.y * HG;
  const int heads = min(HG, H - h0);
  const int rows = min(args.BR, q_len - q0);
  const int row0 = args.req_q_start[req] + q0;
  const int pos0 = args.req_pos0[req] + q0;
  // (what the MMA warp's loops run over: the same in every lane, and the compiler is told so, see tcgen05.cuh)
  const int last_pos = (int)uniform(pos0 + rows - 1);
  const int k_begin = (int)uniform(args.window > 0 ? max(0, pos0 - args.window + 1) / NK * NK : 0);
  const int num_tiles = (last_pos - k_begin) / NK + 1;
  const int* my_table = args.table + (size_t)req * args.table_stride;
  const int own = OWN ? OWN : args.own, chunks = OWN ? OWN + FOREIGN : Dk / 64, foreign = chunks - own, lat_chunks = rank / 64;
  const int own_first = half * own;                    // chunk numbers: latent first, then the rotated part
  const uint32_t s_col = 64u * (uint32_t)own;
  // the i-th foreign chunk's number
  auto foreign_chunk = [&](int i) { return i < own_first ? i : i + own; };

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  if (base & 1023u) {                                  // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicExch(args.error, 58);
    return;
  }
  const uint32_t q_tile = base;                                        // [chunks][128 rows][128 bytes]
  const uint32_t ring = q_tile + (uint32_t)chunks * Q_CHUNK;           // two tiles of [foreign chunks | own chunks], 4 KB each
  const uint32_t p_tile = ring + 2u * (uint32_t)chunks * K_CHUNK;      // [128 rows][64 bytes]
  const uint32_t bars = p_tile + P_BYTES;
  const uint32_t foreign_full = bars, own_full = bars + 16, foreign_empty = bars + 32, own_empty = bars + 48, s_full = bars + 64,
                 s_free = bars + 80, p_full = bars + 96, o_done = bars + 104, tmem_slot = bars + 112;
  volatile uint32_t* tmem_slot_ptr = (volatile uint32_t*)(smem_raw + (tmem_slot - base));

  const int warp = warp_number(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(foreign_full + 8 * b, 1); mbar_init(own_full + 8 * b, 1);
      mbar_init(foreign_empty + 8 * b, 1); mbar_init(own_empty + 8 * b, 1);
      mbar_init(s_full + 8 * b, 1); mbar_init(s_free + 8 * b, 4);
    }
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_columns(own)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  // The pairs' queries as bfloat16: 16-byte pieces of a pair's row, chunk by chunk, in the 128-byte swizzle.  Pairs that do
  // not exist are zeros.  Warp w takes the pairs w, w + 6, ...; a lane the pieces lane, lane + 32, lane + 64 of each (at
  // most 72), four pairs' loads on their way together (one piece at a time took 26 us a CTA, this 7).
  {
    const int pieces = Dk / 8;
    constexpr int LANE_PIECES = (MAX_CHUNKS * 8 + 31) / 32, WARPS = THREADS / 32;
    for (int p0 = warp; p0 < AQ; p0 += 4 * WARPS) {
      float4 x[4][LANE_PIECES][2];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int pr = p0 + u * WARPS, r = pr / HG, hh = pr - r * HG;
        const bool exists = pr < AQ && r < rows && hh < heads;
        const float4* src = reinterpret_cast<const float4*>(args.query + ((size_t)(row0 + (exists ? r : 0)) * H + h0 + (exists ? hh : 0)) * Dk);
#pragma unroll
        for (int j = 0; j < LANE_PIECES; ++j) {
          const int piece = lane + 32 * j;
          x[u][j][0] = x[u][j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (exists && piece < pieces) {
            x[u][j][0] = src[2 * piece];               // (not __ldg: it must not move ahead of the wait above)
            x[u][j][1] = src[2 * piece + 1];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int pr = p0 + u * WARPS;
#pragma unroll
        for (int j = 0; j < LANE_PIECES; ++j) {
          const int piece = lane + 32 * j;
          const float4 a = x[u][j][0], b = x[u][j][1];
          const uint32_t at = (uint32_t)(piece >> 3) * Q_CHUNK + (uint32_t)pr * 128u + (uint32_t)(((piece & 7) ^ (pr & 7)) << 4);
          if (pr < AQ && piece < pieces)
            *reinterpret_cast<uint4*>(smem_raw + at) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the tensor core reads them through the async proxy
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = uniform(*tmem_slot_ptr);

  if (warp == 4) {
    // ---- producer: box = min(page, 32) positions x 64 numbers; lane l brings boxes l, l + 32, ... of a part of the tile
    const int box = min(NK, 1 << args.page_shift), boxes = NK / box;
    const uint32_t box_bytes = (uint32_t)box * 128u;
    const int mine = lane % boxes;                     // this lane's box of every chunk it brings (32 is a multiple of boxes)
    auto row_of = [&](int t) -> int {                  // first row of that box in the pages
      const int kp = k_begin + t * NK + mine * box;
      const int logical = kp >> args.page_shift;
      const int page = (kp <= last_pos && logical < args.table_stride) ? my_table[logical] : 0;
      // a position on no page (one that a window has passed) has weight 0, but what is copied for it enters P C all the
      // same and has to be finite: zeros from behind the pages' end, not the padding page's contents
      return page > 0 ? (page << args.page_shift) + (kp & ((1 << args.page_shift) - 1)) : args.rows_end;
    };
    auto bring = [&](int t, int row, bool owned) -> bool {
      const int b = t & 1;
      const uint32_t full = (owned ? own_full : foreign_full) + 8 * b, empty = (owned ? own_empty : foreign_empty) + 8 * b;
      const int n = owned ? own : foreign;
      bool fine = true;
      if (lane == 0) {
        if (t >= 2) fine = mbar_wait(empty, (uint32_t)((t >> 1) & 1) ^ 1u, args.error, 51);
        if (fine) mbar_expect_tx(full, (uint32_t)n * K_CHUNK);
      }
      fine = __shfl_sync(0xffffffffu, fine ? 1 : 0, 0) != 0;
      if (fine) {
        const uint32_t to = ring + (uint32_t)(b * chunks + (owned ? foreign : 0)) * K_CHUNK;
        for (int i = lane; i < n * boxes; i += 32) {
          const int c = i / boxes, number = owned ? own_first + c : foreign_chunk(c);
          const uint32_t dst = to + (uint32_t)c * K_CHUNK + (uint32_t)mine * box_bytes;
          if (number < lat_chunks) tma_load_2d(dst, &map_latent, number * 64, row, full);
          else tma_load_2d(dst, &map_rope, (number - lat_chunks) * 64, row, full);
        }
      }
      return fine;
    };
    bool ok = true;
    int foreign_issued = 0, own_issued = 0;
    int row = row_of(0);
    for (int t = 0; t < num_tiles && ok; ++t) {
      const int next = t + 1 < num_tiles ? row_of(t + 1) : 0;
      if (foreign > 0) ok = bring(t, row, false);
      if (!ok) break;
      foreign_issued = t + 1;
      ok = bring(t, row, true);
      if (ok) own_issued = t + 1;
      row = next;
    }
    if (!ok && lane == 0) {                            // nobody may be consuming any more: wait for the copies in flight
      for (int t = max(0, foreign_issued - 2); foreign > 0 && t < foreign_issued; ++t) mbar_wait(foreign_full + 8 * (t & 1), (uint32_t)(t >> 1) & 1u, args.error, 52);
      for (int t = max(0, own_issued - 2); t < own_issued; ++t) mbar_wait(own_full + 8 * (t & 1), (uint32_t)(t >> 1) & 1u, args.error, 52);
    }
    __syncwarp();
  } else if (warp == 5) {
    // ---- MMA issue.  The whole warp goes along (the last tile's dead keys are wiped by all its lanes), one lane issues.
    constexpr uint32_t IDESC_S = make_idesc(AQ, NK, 0), IDESC_O = make_idesc(AQ, 64, 1);
    auto wait = [&](uint32_t bar, uint32_t parity, int code) -> bool {           // one answer for the whole warp
      bool fine = true;
      if (lane == 0) fine = mbar_wait(bar, parity, args.error, code);
      return __all_sync(0xffffffffu, fine);
    };
    const bool late = foreign < 4;                     // few foreign chunks: P C waits behind all of the next tile's S
    auto scores = [&](int t, auto which) -> bool {
      constexpr bool owned = decltype(which)::value;
      const int b = t & 1, n = owned ? own : foreign;
      if (n == 0) return true;
      if (!wait((owned ? own_full : foreign_full) + 8 * b, (uint32_t)(t >> 1) & 1u, 53)) return false;
      const bool opens = !owned || foreign == 0;       // the part that starts the tile's sums
      if (opens && t >= 2 && !wait(s_free + 8 * b, (uint32_t)((t >> 1) & 1) ^ 1u, 54)) return false;
      const uint32_t from = ring + (uint32_t)(b * chunks + (owned ? foreign : 0)) * K_CHUNK;
      if (owned && k_begin + t * NK + NK - 1 > last_pos) {
        // Positions past the last row's are nobody's yet: whatever their place in the page holds enters P C times zero, so
        // it has to be finite.  (Their scores are thrown away.)
        const int live = last_pos - (k_begin + t * NK) + 1;
        uint8_t* at = smem_raw + (from - base);
        for (int i = lane; i < n * (NK - live) * 8; i += 32) {
          const int c = i / ((NK - live) * 8), rest = i - c * ((NK - live) * 8);
          *reinterpret_cast<uint4*>(at + c * K_CHUNK + (live + (rest >> 3)) * 128 + (rest & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      __syncwarp();
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < n; ++c) {
          const int number = owned ? own_first + c : foreign_chunk(c);
          const uint64_t da = make_desc(q_tile + (uint32_t)number * Q_CHUNK), db = make_desc(from + (uint32_t)c * K_CHUNK);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma(tmem + s_col + 32u * b, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), IDESC_S, (opens && c == 0 && k == 0) ? 0u : 1u);
        }
        if (!owned) umma_commit(foreign_empty + 8 * b);
        else umma_commit(s_full + 8 * b);
      }
      __syncwarp();
      return true;
    };
    auto weigh = [&](int t) -> bool {                  // O += P C of tile t
      const int b = t & 1;
      if (!wait(p_full, (uint32_t)t & 1u, 55)) return false;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t from = ring + (uint32_t)(b * chunks + foreign) * K_CHUNK;
#pragma unroll
        for (int k = 0; k < NK / 16; ++k) {
          const uint64_t da = make_desc_64(p_tile) + (uint64_t)(2 * k);
#pragma unroll
          for (int c = 0; c < own; ++c)
            umma(tmem + 64u * c, da, make_desc(from + (uint32_t)c * K_CHUNK + (uint32_t)k * 2048u), IDESC_O, (t > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(own_empty + 8 * b);
        umma_commit(o_done);
      }
      __syncwarp();
      return true;
    };
    const std::false_type not_own;
    const std::true_type its_own;
    bool ok = scores(0, not_own) && scores(0, its_own);
    for (int t = 0; t < num_tiles && ok; ++t) {
      const bool more = t + 1 < num_tiles;
      if (more) ok = scores(t + 1, not_own) && (!late || scores(t + 1, its_own));
      if (ok) ok = weigh(t);
      if (ok && more && !late) ok = scores(t + 1, its_own);
    }
  } else {
    // ---- softmax: TMEM lane = pair
    const int pr = threadIdx.x;
    const int r = pr / HG, hh = pr - r * HG;
    const bool exists = r < rows && hh < heads;
    const int qpos = exists ? pos0 + r : -1;           // a pair that does not exist sees nothing
    const int qlow = args.window > 0 ? qpos - args.window : -1;        // the last position out of its sight
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    uint8_t* p_row = smem_raw + (p_tile - base) + pr * 64;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    auto cached = [&](int t) -> unsigned {             // bit j: position j of tile t is on a page
      const int kp = k_begin + t * NK + lane;
      const int page = (t < num_tiles && kp <= last_pos) ? my_table[kp >> args.page_shift] : 0;
      return __ballot_sync(0xffffffffu, page > 0);
    };
    unsigned there = cached(0);
    for (int t = 0; t < num_tiles; ++t) {
      const int b = t & 1, k0 = k_begin + t * NK;
      const unsigned there_next = cached(t + 1);
      if (lane == 0) ok = mbar_wait(s_full + 8 * b, (uint32_t)(t >> 1) & 1u, args.error, 56);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      tc_fence_after();
      uint32_t s[32];
      tmem_ld32(tmem + s_col + 32u * b + lane_addr, s);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free + 8 * b);
      // the keys that this pair sees
      const int up = qpos - k0, low = qlow - k0;       // visible: low < j <= up
      unsigned seen = up >= 31 ? 0xffffffffu : (up < 0 ? 0u : (2u << up) - 1u);
      if (low >= 0) seen &= low >= 31 ? 0u : ~((2u << low) - 1u);
      seen &= there;
      there = there_next;
      float m_tile = -INFINITY;
      if (__all_sync(0xffffffffu, seen == 0xffffffffu)) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float x = __uint_as_float(s[j]) * args.scale_log2;
          s[j] = __float_as_uint(x);
          m_tile = fmaxf(m_tile, x);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float x = (seen >> j) & 1u ? __uint_as_float(s[j]) * args.scale_log2 : -INFINITY;
          s[j] = __float_as_uint(x);
          m_tile = fmaxf(m_tile, x);
        }
      }
      const bool move = m_tile > m_used;               // minus infinity at first: any visible key moves it
      // P's place is free, and O is at rest, when the tile before has been summed
      if (t > 0) {
        if (lane == 0) ok = mbar_wait(o_done, (uint32_t)(t - 1) & 1u, args.error, 57);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
      }
      if (__any_sync(0xffffffffu, move)) {
        const float m_new = move ? m_tile : m_used;
        const float alpha = move ? exp2f(m_used - m_new) : 1.f;        // exp2(-inf) = 0 before the first visible key
        m_used = m_new;
        l *= alpha;
        if (t > 0) {
          tc_fence_after();
          for (int c = 0; c < own * 64; c += 32) {
            uint32_t o[32];
            tmem_ld32(tmem + (uint32_t)c + lane_addr, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tmem_st32(tmem + (uint32_t)c + lane_addr, o);
          }
          tmem_st_wait();
        }
      }
      const float m = m_used == -INFINITY ? 0.f : m_used;
#pragma unroll
      for (int piece = 0; piece < 4; ++piece) {
        float p[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          p[j] = exp2f(__uint_as_float(s[piece * 8 + j]) - m);
          l += p[j];
        }
        *reinterpret_cast<uint4*>(p_row + ((piece ^ ((pr >> 1) & 3)) << 4)) =
            make_uint4(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]), pack_bf16(p[4], p[5]), pack_bf16(p[6], p[7]));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok) {
      if (lane == 0) ok = mbar_wait(o_done, (uint32_t)(num_tiles - 1) & 1u, args.error, 57);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    }
    if (ok) {
      // O out: through the queries' place in shared memory (every product is done), so that a warp stores 128 bytes of a
      // row at a time
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      float* stage = reinterpret_cast<float*>(smem_raw) + warp * 32 * 36;
      for (int c = 0; c < own * 64; c += 32) {
        uint32_t o[32];
        tmem_ld32(tmem + (uint32_t)c + lane_addr, o);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(stage + lane * 36 + j) = make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv,
                                                                          __uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int at = i * 4 + (lane >> 3), pair = warp * 32 + at;
          const int pr_row = pair / HG, pr_head = pair - pr_row * HG;
          const float4 v = *reinterpret_cast<const float4*>(stage + at * 36 + (lane & 7) * 4);
          if (pr_row < rows && pr_head < heads)
            *reinterpret_cast<float4*>(args.out + ((size_t)(row0 + pr_row) * H + h0 + pr_head) * rank + own_first * 64 + c + (lane & 7) * 4) = v;
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_columns(own)) : "memory");
  }
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

// No more CTAs may share a multiprocessor than its 512 tensor-memory columns serve: one more would wait for them until
// another is through, while a multiprocessor beside it has none (measured, latent 256 without a rotated part: 101 requests'
// tiles over 500 keys 125 us, two to a multiprocessor where 62 were to be had).  Shared memory holds them off.
constexpr size_t smem_bytes(int chunks, int own) {
  const size_t used = (size_t)chunks * (Q_CHUNK + 2 * K_CHUNK) + P_BYTES + 128, apart = (228 * 1024) / (512 / tmem_columns(own) + 1) + 128;
  return used > apart ? used : apart;
}

int setup() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (err != cudaSuccess || fn == nullptr || q != cudaDriverEntryPointSuccess)
      return ayk_fail("ayk_latent_attention_tc: cuTensorMapEncodeTiled is not available from this driver");
    g_encode = (EncodeTiledFn)fn;
  }
  if (!g_error_host) {
    cudaError_t err = cudaHostAlloc((void**)&g_error_host, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    if (err != cudaSuccess) return ayk_fail("ayk_latent_attention_tc: cudaHostAlloc: %s", cudaGetErrorString(err));
    *g_error_host = 0;
    err = cudaHostGetDevicePointer((void**)&g_error_dev, g_error_host, 0);
    if (err != cudaSuccess) return ayk_fail("ayk_latent_attention_tc: cudaHostGetDevicePointer: %s", cudaGetErrorString(err));
  }
  if (!g_configured.here()) {
    cudaError_t err = cudaFuncSetAttribute(latent_tc_kernel<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(MAX_CHUNKS, 4));
    if (err == cudaSuccess) err = cudaFuncSetAttribute(latent_tc_kernel<5, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(9, 4));
    if (err == cudaSuccess) err = cudaFuncSetAttribute(latent_tc_kernel<4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(8, 4));
    if (err != cudaSuccess) return ayk_fail("ayk_latent_attention_tc: shared memory %zu: %s", smem_bytes(MAX_CHUNKS, 4), cudaGetErrorString(err));
    g_configured.here() = true;
  }
  return 0;
}

// rows x width bfloat16; box of `box` rows x 64 numbers, 128-byte swizzle.
int encode(CUtensorMap* map, const void* ptr, long long rows, int width, int box_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)width * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return ayk_fail("ayk_latent_attention_tc: cuTensorMapEncodeTiled failed with %d (rows %lld, width %d)", (int)r, rows, width);
  return 0;
}

}  // namespace

AYK_EXPORT int ayk_latent_tc_error() { return g_error_host ? *g_error_host : 0; }

// Whether the tcgen05 kernel takes this geometry: keys in whole chunks of 64 numbers, at most nine; latents beyond 256 in two
// equal halves of whole chunks; pages of at least the swizzle's 8 rows.
AYK_EXPORT int ayk_latent_attention_tc_takes(int rank, int rot, int pages, int page_size, const void* query, const void* latent_pages, const void* rope_pages) {
  if (rank < 64 || rank % 64 != 0 || rank > 512 || (rank > 256 && rank % 128 != 0) || rot < 0 || rot % 64 != 0 || rank + rot > 64 * MAX_CHUNKS) return 0;
  if (page_size < 8 || (page_size & (page_size - 1)) != 0 || (long long)pages * page_size >= (1ll << 31)) return 0;
  return (uintptr_t)query % 16 == 0 && (uintptr_t)latent_pages % 16 == 0 && (uintptr_t)rope_pages % 16 == 0;
}

// As ayk_latent_attention, bfloat16 pages [pages, page_size, rank] and [pages, page_size, rot], any rows per request.
AYK_EXPORT int ayk_latent_attention_tc(float* out, const float* query, const void* latent_pages, const void* rope_pages, int pages,
                                       const int* table, int table_stride, const int* req_q_start, const int* req_pos0, int num_req,
                                       int total_rows, int H, int rank, int rot, int page_size, float scale, int window,
                                       cudaStream_t stream) {
  if (num_req == 0 || total_rows == 0) return 0;
  AYK_REQUIRE(ayk_latent_attention_tc_takes(rank, rot, pages, page_size, query, latent_pages, rope_pages) && (uintptr_t)out % 16 == 0,
              "ayk_latent_attention_tc: latent %d + %d, pages of %d, or the operands' alignment, are not taken", rank, rot, page_size);
  AYK_REQUIRE(H >= 1, "ayk_latent_attention_tc: %d heads", H);
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (setup() != 0) return -1;
  }
  int shift = 0;
  while ((1 << shift) < page_size) ++shift;
  const int box = page_size < NK ? page_size : NK;
  CUtensorMap ml, mr;
  if (encode(&ml, latent_pages, (long long)pages * page_size, rank, box) != 0) return -1;
  if (rot > 0) { if (encode(&mr, rope_pages, (long long)pages * page_size, rot, box) != 0) return -1; }
  else mr = ml;
  const int HG = H < AQ ? H : AQ, BR = AQ / HG, halves = rank > 256 ? 2 : 1;
  // the halves of a tile side by side (they read the same keys); tiles along x, where a grid has room for any step's rows
  dim3 grid((unsigned)halves * (unsigned)(total_rows / BR + num_req), (H + HG - 1) / HG);
  AYK_REQUIRE(grid.y <= 65535, "ayk_latent_attention_tc: %d heads", H);
  LatentArgs args{out, query, table, req_q_start, req_pos0, g_error_dev, table_stride, num_req, H, HG, BR, rank, rot, shift, window,
                  rank / 64 / halves, pages * page_size, halves - 1, scale * 1.4426950408889634f};
  const size_t smem = smem_bytes((rank + rot) / 64, rank / 64 / halves);
  if (rank == 512 && rot == 64) ayk_launch(latent_tc_kernel<5, 4>, grid, dim3(THREADS), smem, stream, ml, mr, args);
  else if (rank == 512 && rot == 0) ayk_launch(latent_tc_kernel<4, 4>, grid, dim3(THREADS), smem, stream, ml, mr, args);
  else ayk_launch(latent_tc_kernel<0, 0>, grid, dim3(THREADS), smem, stream, ml, mr, args);
  return ayk_check_launch("ayk_latent_attention_tc");
}
