// Causal attention of a step's rows over the paged cache, any mix of prompt
// portions and single decoded tokens, on the FP32 pipes.  It is the attention
// of the true 32-bit path and the general fallback for head sizes and options
// that the faster kernels refuse.
//
// Formula (kernel/triton/paged_attention.py:295-355): for the query at absolute
// position p of a request, s_j = (q . k_j) * scale over the cached positions
// j <= p of that request (and j > p - window when a window is given), online
// softmax with running maximum and sum in 32-bit, o = sum_j a_j v_j; a query
// with no visible key gives 0.  The keys and values of the step's own rows are
// already in the cache (ayk_kv_append runs first, as attention/base.py:67-69
// stores before it attends).
//
// One block works on up to 32 consecutive rows of one request and one head.  Keys and values are taken KT at a
// time (64, or 32 for heads wider than 128): the float32 cache is copied by cp.async a tile ahead, a warp looking up
// its keys' cells once per tile; bfloat16 is widened on the way in.  A thread owns 4 rows: KT / 16 scores of each, four
// head-dim columns of each per 64 of the head size; scores and the weighted sum are register tiles fed with float4 (64
// products per 8 reads of shared memory).  Only the running maximum crosses threads in a tile, sums do at the end.  Warps
// without a live row only copy.
//
// Bound by latency per key tile when rows are few and by shared memory when they are many.  Before, a key tile of 32 cost
// 20 us (a division, a block-table look-up and a 4-byte load per element, nothing ahead): GPT-2 small, 372 prompt rows
// beside 5 single ones, 12 heads: 132 us, now 30.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int BQ = 32;       // rows per block
constexpr int WARPS = 4;
constexpr int MAX_DH = 256;

__host__ __device__ constexpr int tile_keys(int nc) { return nc <= 2 ? 64 : 32; }
// Floats per row of a tile: whole 16-byte pieces, an odd number of them, so that eight neighbouring rows' pieces lie on different banks.
__host__ __device__ inline int row_floats(int Dh) { return (((Dh + 3) / 4) | 1) * 4; }
size_t smem_floats(int Dh, int KT) {
  return (size_t)BQ * row_floats(Dh) + (size_t)4 * KT * row_floats(Dh) + (size_t)BQ * (KT + 4) + (size_t)2 * KT;
}

__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// NC: head-dim columns in runs of 64.
template <typename T, int NC>
__global__ void __launch_bounds__(WARPS * 32)
attention_simt_kernel(T* __restrict__ out, const T* q, int q_stride,
                      const T* kcache, const T* vcache,
                      const int* __restrict__ table, int table_stride,
                      const int* __restrict__ req_q_start, const int* __restrict__ req_pos0,
                      int num_req, int H, int Hkv, int Dh, int page_size, float scale, int window) {
  constexpr int KT = tile_keys(NC), KJ = KT / 16, LDP = KT + 4;
  if (gridDim.x * gridDim.y <= AYK_FEW_BLOCKS) pdl_trigger();
  pdl_wait();
  // Which request and which of its row tiles is this block?
  int tile = blockIdx.x, req = -1, q0 = 0, q_len = 0;
  for (int r = 0; r < num_req; ++r) {
    int len = req_q_start[r + 1] - req_q_start[r];
    int tiles = (len + BQ - 1) / BQ;
    if (tile < tiles) { req = r; q0 = tile * BQ; q_len = len; break; }
    tile -= tiles;
  }
  if (req < 0) return;
  const int h = blockIdx.y, kvh = h / (H / Hkv);
  const int rows = min(BQ, q_len - q0);
  const int row0 = req_q_start[req] + q0;       // first global row of the tile
  const int pos0 = req_pos0[req] + q0;          // its absolute position
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;      // keys tx + 16 j, columns 4 tx + 64 c; rows 4 ty + i
  const int LD = row_floats(Dh), D4 = (Dh + 3) / 4;

  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                    // [BQ][LD]
  float* Ks = Qs + BQ * LD;            // two buffers of [KT][LD]
  float* Vs = Ks + 2 * KT * LD;        // two buffers of [KT][LD]
  float* Ps = Vs + 2 * KT * LD;        // [BQ][LDP]
  int* there = reinterpret_cast<int*>(Ps + BQ * LDP);          // per buffer and key: is it cached

  const int last_pos = pos0 + rows - 1;
  int k_begin = 0;
  if (window > 0) k_begin = max(0, pos0 - window + 1) / KT * KT;
  const int* my_table = table + (size_t)req * table_stride;
  constexpr int PER_WARP = KT / WARPS;          // keys of a tile that a warp copies
  const bool vec = Dh % 4 == 0 && ((uintptr_t)kcache | (uintptr_t)vcache) % 16 == 0;

  // Lane j looks up key j of the warp's share of a tile: its cell in the pages, or -1.
  auto lookup = [&](int k0) {
    const int kp = k0 + warp * PER_WARP + lane;
    const int page = (lane < PER_WARP && kp <= last_pos) ? my_table[kp / page_size] : 0;
    return page > 0 ? page * page_size + kp % page_size : -1;
  };
  auto fetch = [&](int cells, int b) {
    if (lane < PER_WARP) there[b * KT + warp * PER_WARP + lane] = cells >= 0;
    for (int j = 0; j < PER_WARP; ++j) {
      const int cell = __shfl_sync(0xffffffffu, cells, j), key = warp * PER_WARP + j;
      float* kd = Ks + (b * KT + key) * LD;
      float* vd = Vs + (b * KT + key) * LD;
      const size_t at = ((size_t)max(cell, 0) * Hkv + kvh) * Dh;
      for (int c = lane; c < 2 * D4; c += 32) {
        const bool of_k = c < D4;
        const int d = (of_k ? c : c - D4) * 4;
        float* dst = (of_k ? kd : vd) + d;
        const T* src = (of_k ? kcache : vcache) + at + d;
        if (cell < 0) {
          *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else if constexpr (sizeof(T) == 4) {
          if (vec) copy16(dst, reinterpret_cast<const float*>(src));
          else
            for (int e = 0; e < 4; ++e) {
              if (d + e < Dh) copy4(dst + e, reinterpret_cast<const float*>(src) + e);
              else dst[e] = 0.f;
            }
        } else {
          for (int e = 0; e < 4; ++e) dst[e] = d + e < Dh ? to_float<T>(src[e]) : 0.f;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  int next = lookup(k_begin);
  fetch(next, 0);
  next = lookup(k_begin + KT);
  for (int i = threadIdx.x; i < BQ * D4 * 4; i += blockDim.x) {
    const int r = i / (D4 * 4), d = i - r * (D4 * 4);
    Qs[r * LD + d] = (r < rows && d < Dh) ? to_float<T>(q[(size_t)(row0 + r) * q_stride + h * Dh + d]) : 0.f;
  }

  float acc[4][NC][4];
  float m_run[4], l_run[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[i][c][0] = acc[i][c][1] = acc[i][c][2] = acc[i][c][3] = 0.f;
  }
  const bool live = warp * 8 < rows;            // this warp's rows 8 warp ... + 7

  int b = 0;
  for (int k0 = k_begin; k0 <= last_pos; k0 += KT, b ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                            // the tile (and Qs) is there; the other buffer has been read
    if (k0 + KT <= last_pos) {
      fetch(next, b ^ 1);
      next = lookup(k0 + 2 * KT);
    }
    if (!live) continue;
    const float* Kt = Ks + b * KT * LD;
    const float* Vt = Vs + b * KT * LD;
    float s[4][KJ];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < KJ; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D4; ++d) {
      float4 qv[4], kv[KJ];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(Qs + (ty * 4 + i) * LD + d * 4);
#pragma unroll
      for (int j = 0; j < KJ; ++j) kv[j] = *reinterpret_cast<const float4*>(Kt + (tx + 16 * j) * LD + d * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < KJ; ++j) {
          s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
          s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
          s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
        }
    }
    int cached[KJ];
#pragma unroll
    for (int j = 0; j < KJ; ++j) cached[j] = there[b * KT + tx + 16 * j];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int qpos = pos0 + ty * 4 + i;
      float m_new = m_run[i];
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const int kp = k0 + tx + 16 * j;
        const bool valid = cached[j] && kp <= qpos && (window <= 0 || kp > qpos - window);
        s[i][j] = valid ? s[i][j] * scale : -INFINITY;
        m_new = fmaxf(m_new, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));      // the 16 threads of a row
      const float m_use = m_new > -INFINITY ? m_new : 0.f;
      const float alpha = expf(m_run[i] - m_use);          // exp(-inf) = 0 before the first visible key
      m_run[i] = m_new;
      l_run[i] *= alpha;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const float p = expf(s[i][j] - m_use);             // 0 where the key is out of sight
        l_run[i] += p;
        Ps[(ty * 4 + i) * LDP + tx + 16 * j] = p;
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) { acc[i][c][0] *= alpha; acc[i][c][1] *= alpha; acc[i][c][2] *= alpha; acc[i][c][3] *= alpha; }
    }
    __syncwarp();                               // a warp reads the weights of its own rows only
#pragma unroll 2
    for (int k = 0; k < KT; k += 4) {
      float4 p[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(Ps + (ty * 4 + i) * LDP + k);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int d = 4 * tx + 64 * c;
        if (NC > 1 && d >= D4 * 4) continue;
        const int col = NC > 1 ? d : min(d, D4 * 4 - 4);          // heads below 64: columns that do not exist are read and not stored
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(Vt + (k + u) * LD + col);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float w[4] = {p[i].x, p[i].y, p[i].z, p[i].w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[i][c][0] = fmaf(w[u], v[u].x, acc[i][c][0]);
            acc[i][c][1] = fmaf(w[u], v[u].y, acc[i][c][1]);
            acc[i][c][2] = fmaf(w[u], v[u].z, acc[i][c][2]);
            acc[i][c][3] = fmaf(w[u], v[u].w, acc[i][c][3]);
          }
        }
      }
    }
    __syncwarp();
  }
  if (!live) return;

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = ty * 4 + i;
    float l = l_run[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (row >= rows) continue;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    T* o = out + (size_t)(row0 + row) * ((size_t)H * Dh) + h * Dh;
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = 4 * tx + 64 * c + e;
        if (d < Dh) o[d] = from_float<T>(acc[i][c][e] * inv);
      }
  }
}

template <typename T, int NC>
int launch(void* out, const void* q, int q_stride, const void* kcache, const void* vcache, const int* table, int table_stride,
           const int* req_q_start, const int* req_pos0, int num_req, int total_rows, int H, int Hkv, int Dh, int page_size, float scale,
           int window, cudaStream_t stream) {
  const size_t smem = smem_floats(Dh, tile_keys(NC)) * sizeof(float);
  static AykPerDevice configured;
  bool& done = configured.here();
  if (!done) {                                  // the largest size that this copy is launched with
    const size_t most = smem_floats(NC * 64, tile_keys(NC)) * sizeof(float);
    cudaError_t err = cudaFuncSetAttribute(attention_simt_kernel<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (err != cudaSuccess) return ayk_fail("ayk_attention_simt: shared memory %zu: %s", most, cudaGetErrorString(err));
    done = true;
  }
  dim3 grid(total_rows / BQ + num_req, H);      // the sum of ceil(len / BQ) never exceeds this
  ayk_launch_as(grid.x * grid.y <= AYK_FEW_BLOCKS, attention_simt_kernel<T, NC>, grid, dim3(WARPS * 32), smem, stream, (T*)out, (const T*)q,
                q_stride, (const T*)kcache, (const T*)vcache, table, table_stride, req_q_start, req_pos0, num_req, H, Hkv, Dh,
                page_size, scale, window);
  return ayk_check_launch("ayk_attention_simt");
}

}  // namespace

AYK_EXPORT int ayk_attention_tile_rows() { return BQ; }

// out[T, H*Dh]; q rows of q_stride elements (head h at offset h*Dh); caches
// [pages, page_size, Hkv, Dh]; table[num_req, table_stride]; req_q_start[num_req+1]
// row offsets of each request's rows; req_pos0[num_req] absolute position of a
// request's first row.  total_rows = req_q_start[num_req] (known to the host).
AYK_EXPORT int ayk_attention_simt(void* out, const void* q, int q_stride, const void* kcache,
                                  const void* vcache, const int* table, int table_stride,
                                  const int* req_q_start, const int* req_pos0, int num_req,
                                  int total_rows, int H, int Hkv, int Dh, int page_size, float scale,
                                  int window, int dtype, cudaStream_t stream) {
  if (num_req == 0 || total_rows == 0) return 0;
  AYK_REQUIRE(Dh >= 1 && Dh <= MAX_DH, "ayk_attention_simt: head size %d is not in [1, %d]", Dh, MAX_DH);
  AYK_REQUIRE(Hkv >= 1 && H % Hkv == 0, "ayk_attention_simt: %d heads cannot share %d key/value heads", H, Hkv);
  AYK_REQUIRE(H <= 65535, "ayk_attention_simt: too many heads (%d)", H);
#define AYK_SIMT(T)                                                                                                              \
  switch ((Dh + 63) / 64) {                                                                                                     \
    case 1: return launch<T, 1>(out, q, q_stride, kcache, vcache, table, table_stride, req_q_start, req_pos0, num_req, total_rows, H, \
                                Hkv, Dh, page_size, scale, window, stream);                                                      \
    case 2: return launch<T, 2>(out, q, q_stride, kcache, vcache, table, table_stride, req_q_start, req_pos0, num_req, total_rows, H, \
                                Hkv, Dh, page_size, scale, window, stream);                                                      \
    case 3: return launch<T, 3>(out, q, q_stride, kcache, vcache, table, table_stride, req_q_start, req_pos0, num_req, total_rows, H, \
                                Hkv, Dh, page_size, scale, window, stream);                                                      \
    default: return launch<T, 4>(out, q, q_stride, kcache, vcache, table, table_stride, req_q_start, req_pos0, num_req, total_rows, H, \
                                 Hkv, Dh, page_size, scale, window, stream);                                                     \
  }
  if (dtype == AYK_DTYPE_F32) { AYK_SIMT(float) }
  if (dtype == AYK_DTYPE_BF16) { AYK_SIMT(__nv_bfloat16) }
#undef AYK_SIMT
  return ayk_fail("ayk_attention_simt: unknown dtype %d", dtype);
}
